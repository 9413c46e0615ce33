"""FP32 short-range kernels of the differentiable mode (diff_rows.cu): every
instantiation (8 or 16 slots; no, 2 or 8 min/max slots; with and without
directional factors and desolvation terms) on boxes that cut bricks and warps.

Forward: the parity bar against the FP64 oracle.  Adjoint: against the FP64
twin, whose per-pair code is separate.  An FP32 distance is off by at most
about 4 * 2^-24 relative, 5e-4 bins at 8 A, so about one pair in a thousand
takes the neighbouring bin's slope; slopes of neighbouring bins differ by far
less than themselves except next to a table's clamp, and 1e-3 of the gradient's
norm bounds what those pairs add.
"""
import numpy as np
import pytest

from conftest import make_case, tolerance_ok

pytestmark = pytest.mark.gpu

SETS = {
    "plain_small": dict(ligand_types=["C", "A", "N"]),
    "plain_16": dict(ligand_types=["C", "A", "N", "S", "P", "F", "Cl", "Br", "I"]),
    "ad4_8": dict(ligand_types=["A", "C", "HD", "N", "NA", "OA"]),
    "ad4_16": dict(ligand_types=["A", "C", "HD", "N", "NA", "OA", "SA", "S", "P", "F"]),
    "three_minmax": dict(ligand_types=["HD", "HS", "NA", "OA", "C"]),
    "disorder": dict(ligand_types=["HD", "NA", "OA", "C"], pre_lines=["disorder_h"]),
    "no_dsolv": dict(ligand_types=["OA", "C"], dsolvmap=False, elecmap=False),
    "vina": dict(ligand_types=["A", "C", "HD", "N", "NA", "OA"]),
}


@pytest.mark.parametrize("npts", [(2, 2, 2), (8, 6, 4), (18, 10, 14)])
@pytest.mark.parametrize("name", list(SETS))
def test_rows_forward_and_adjoint(tmp_path, gpu_ctx, name, npts):
    from autogrid_b200 import Diff
    from oracle.oracle import oracle_points_lin
    job, prob = make_case(tmp_path, name, 350, npts, seed=sum(npts), radius=10.0, **SETS[name])
    if name == "vina":
        prob = job.vina_problem()
    w = np.random.default_rng(1).normal(size=prob.map_shape)
    d64, d32 = Diff(gpu_ctx, prob, "fp64"), Diff(gpu_ctx, prob, "fp32")
    for d in (d64, d32):
        d.forward()
    ref = oracle_points_lin(prob, closest_h=d64.closest_h() if name != "vina" else None)
    got = d32.maps().reshape(prob.n_maps, -1).astype(np.float64)
    assert tolerance_ok(got, ref).all()
    g64, g32 = d64.backward(w), d32.backward(w.astype(np.float32))
    for key in ("coord", "charge"):
        err, norm = np.linalg.norm(g32[key] - g64[key]), np.linalg.norm(g64[key])
        assert err <= 1e-3 * norm, f"{key}: {err / max(norm, 1e-300):.2g}"
    d32.close(); d64.close()
