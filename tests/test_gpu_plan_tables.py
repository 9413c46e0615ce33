"""One-shot calls pack the kernels' tables on the GPU and send their inputs in
one image of the context; plans pack on the host in memory of their own.  Both
run the same kernels in the same order on boxes of one z slab, so their maps
agree in every bit: for tables of one, a few and many maps (rows of 8 columns,
a part of one, several groups), both dielectrics, and calls of changing size
through one context, whose image grows and is used again.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu

LIGANDS = {1: ["C"], 3: ["HD", "OA", "N"], 9: ["C", "A", "HD", "OA", "N", "NA", "SA", "S", "F"],
           17: ["C", "A", "HD", "OA", "N", "NA", "SA", "S", "F", "H", "Cl", "Br", "I", "P", "Zn", "Fe", "Mg"]}


@pytest.mark.parametrize("dielectric", [-0.1465, 40.0])
def test_one_shot_equals_plan(tmp_path, gpu_ctx, dielectric):
    for k, (n_atoms, n_types) in enumerate([(60, 1), (700, 9), (33, 3), (1500, 17), (700, 1)]):
        path = tmp_path / str(k)
        path.mkdir()
        _, prob = make_case(path, "tab", n_atoms, (14, 10, 8), seed=k, ligand_types=LIGANDS[n_types],
                            dielectric=dielectric)
        got = gpu_ctx.compute(prob, "fp32")
        plan = gpu_ctx.plan(prob)
        plan.run()
        want = plan.download()
        plan.close()
        assert np.ascontiguousarray(got).tobytes() == np.ascontiguousarray(want).tobytes(), (n_atoms, n_types)
