"""Order of staged candidates by receptor type, on the CPU.

tests/native/type_sort_check.cpp runs the kernels' counting sort
(autogrid_b200/csrc/kernels/type_sort.cuh) with a host thread per GPU thread,
whose stores reach other threads only at barriers and there in random order: a
missing barrier gives wrong places.
"""
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    out = tmp_path_factory.mktemp("tsc") / "type_sort_check"
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-Wno-unknown-pragmas", "-I",
                        str(ROOT / "autogrid_b200" / "csrc"), str(ROOT / "tests" / "native" / "type_sort_check.cpp"),
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_places_are_those_of_a_stable_sort(checker, seed):
    r = subprocess.run([str(checker), str(seed)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
