"""Differentiable mode in FP32: a map without weight in the loss leaves the
gradient alone, also where its table holds values that are not finite, and so
does the weight of a covalent map, which no atom enters.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu

SETS = {  # 8 and 16 slots, with and without directional factors and desolvation terms
    "plain": dict(ligand_types=["C", "A", "N"]),
    "plain_16": dict(ligand_types=["C", "A", "N", "S", "P", "F", "Cl", "Br", "I"]),
    "ad4_8": dict(ligand_types=["C", "HD", "NA", "OA"]),
    "ad4_16": dict(ligand_types=["A", "C", "HD", "N", "NA", "OA", "SA", "S", "P", "F"]),
    "vina": dict(ligand_types=["C", "A", "N"]),
}


def gradient(gpu_ctx, prob, w):
    from autogrid_b200 import Diff
    d = Diff(gpu_ctx, prob, "fp32")
    d.forward()
    g = d.backward(w)
    d.close()
    return g


def same(got, ref):
    for key, v in ref.items():
        # the sums' order differs from run to run (FP64 atomics)
        assert np.linalg.norm(got[key] - v) <= 1e-9 * np.linalg.norm(v) + 1e-12, key


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("bins", [slice(0, 1024), slice(300, 400), slice(1023, 1024)])
@pytest.mark.parametrize("name", list(SETS))
def test_unweighted_map_with_values_not_finite(tmp_path, gpu_ctx, name, bins, value):
    job, prob = make_case(tmp_path, name, 300, (10, 8, 6), seed=4, radius=9.0, **SETS[name])
    if name == "vina":
        prob = job.vina_problem()
    w = np.random.default_rng(2).normal(size=prob.map_shape).astype(np.float32)
    nT, nM = max(prob.scalars["n_rec_types"], 1), prob.scalars["n_atom_maps"]
    tables = prob.arrays["e_vdw_hb"][: nT * nM * 1024].reshape(nT, nM, 1024)
    w[1] = 0.0
    ref = gradient(gpu_ctx, prob, w)
    tables[:, 1, bins] = value
    same(gradient(gpu_ctx, prob, w), ref)


def test_weight_of_a_covalent_map(tmp_path, gpu_ctx):
    _, prob = make_case(tmp_path, "cov", 300, (10, 8, 6), seed=4, radius=9.0, ligand_types=["C", "OA", "Z"],
                        extra_lines=["covalentmap 1.5 1000.0 1.0 -1.5 2.0"])
    m = int(np.flatnonzero(prob.arrays["map_is_covalent"])[0])
    w = np.random.default_rng(2).normal(size=prob.map_shape).astype(np.float32)
    ref = gradient(gpu_ctx, prob, w)
    w[m] = np.inf
    same(gradient(gpu_ctx, prob, w), ref)
