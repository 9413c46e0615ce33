"""FP32 near-field kernel (near_rows.cu): both accumulator counts, several
groups of maps, boxes that cut bricks, candidate lists longer than one staged
chunk, spacings whose frame coordinates are no exact floats, against the FP64
oracle with the parity bar; and the FP64 twin on the same problems to 1e-9.
"""
import numpy as np
import pytest

from conftest import make_case, tolerance_ok

pytestmark = pytest.mark.gpu

T14 = ["A", "C", "HD", "N", "NA", "OA", "SA", "S", "P", "F", "Cl", "Br", "I", "Fe"]
CASES = {
    "27_points": dict(n_atoms=200, npts=(2, 2, 2), ligand_types=["C", "HD"]),
    "cut_bricks_8": dict(n_atoms=600, npts=(8, 10, 4), ligand_types=["A", "C", "HD", "N", "NA", "OA"]),
    "exact_brick_9_maps": dict(n_atoms=600, npts=(14, 6, 2), ligand_types=T14[:9]),
    "two_groups": dict(n_atoms=500, npts=(10, 8, 6), ligand_types=T14 + ["HS", "NS", "OS", "Mg", "Zn", "Ca"]),
    "three_minmax": dict(n_atoms=500, npts=(6, 12, 8), ligand_types=["HD", "HS", "NA", "C"], pre_lines=["disorder_h"]),
    "coarse_spacing": dict(n_atoms=700, npts=(12, 12, 12), spacing=0.9, ligand_types=["OA", "HD", "C"]),
    "inexact_spacing": dict(n_atoms=700, npts=(16, 10, 12), spacing=0.37, ligand_types=["OA", "NA", "HD", "SA"]),
    "dense": dict(n_atoms=900, npts=(10, 10, 10), radius=10.5, ligand_types=["A", "C", "HD", "N", "NA", "OA"]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_near_maps_against_oracle(tmp_path, gpu_ctx, name):
    from oracle.oracle import oracle_points
    kw = dict(CASES[name])
    n, npts = kw.pop("n_atoms"), kw.pop("npts")
    _, prob = make_case(tmp_path, name, n, npts, seed=n + len(name), radius=kw.pop("radius", None), **kw)
    ref, flags = oracle_points(prob)
    free = flags == 0
    got = gpu_ctx.compute(prob, "fp32").reshape(prob.n_maps, -1)
    assert tolerance_ok(got[:, free], ref[:, free]).all()
    twin = gpu_ctx.compute(prob, "fp64").reshape(prob.n_maps, -1)
    near = [m for m in range(prob.n_maps) if m != prob.scalars["elec_map"]]  # the twin's e map is another kernel's
    np.testing.assert_allclose(twin[near][:, free], ref[near][:, free], rtol=1e-9, atol=1e-9)


@pytest.mark.parametrize("n_atoms,npts,spacing", [(60, (18, 18, 16), 1.0), (25, (30, 6, 8), 1.3)])
def test_points_without_a_hydrogen_in_reach(tmp_path, gpu_ctx, n_atoms, npts, spacing):
    """Boxes larger than the receptor: points with no DS/D1 atom within 8 A (the
    reference takes one further away, which no pair in range reads), bricks with
    such atoms for a part of their points, and bricks without any atom."""
    from oracle.oracle import oracle_points
    _, prob = make_case(tmp_path, "far_h", n_atoms, npts, seed=n_atoms, spacing=spacing,
                        ligand_types=["A", "C", "HD", "N", "NA", "OA"])
    a = prob.arrays
    h = np.isin(a["hbond"], (1, 2))
    ax = [(np.arange(n) - (n - 1) // 2) * spacing for n in prob.n1]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r2 = ((a["coord"].reshape(-1, 3)[h][:, None] - np.stack([x, y, z], -1).reshape(-1, 3)) ** 2).sum(-1).min(0)
    assert (r2 > 64).any() and (r2 < 64).any()
    ref, flags = oracle_points(prob)
    free = flags == 0
    got = gpu_ctx.compute(prob, "fp32").reshape(prob.n_maps, -1)
    assert tolerance_ok(got[:, free], ref[:, free]).all()
    twin = gpu_ctx.compute(prob, "fp64").reshape(prob.n_maps, -1)
    near = [m for m in range(prob.n_maps) if m != prob.scalars["elec_map"]]
    np.testing.assert_allclose(twin[near][:, free], ref[near][:, free], rtol=1e-9, atol=1e-9)
