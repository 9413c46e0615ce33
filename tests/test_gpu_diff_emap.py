"""FP32 e map of the differentiable mode (diff_emap_rows.cu): boxes that cut
its 32x8x8 frames, atom counts around its 32-atom runs and chunks, atoms on
grid points and within 0.5 A of them, distances past the last table bin, and
several conformers, against the FP64 twin (itself checked against the oracle).

A sum has runs of at most 256 terms: the forward's rounding stays below
255 + 10 units of 2^-24 of the sum of the terms' magnitudes.  The adjoint may
take a neighbouring bin's slope for about one pair in a thousand; slopes of
neighbouring bins of this table differ by 1e-3 of themselves, so 1e-4 of the
norm bounds that and the rounding of the sums.  The atom on a grid point is not
in that comparison: its distances to the points of the axes lie on bin edges,
where the interpolated map has no derivative.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [(2, 2, 2), (30, 8, 6), (32, 10, 8), (40, 16, 18)])
@pytest.mark.parametrize("n_atoms,radius,conformers", [(20, None, 1), (65, 110.0, 2), (300, None, 1), (700, None, 3)])
def test_e_map_and_adjoint(tmp_path, gpu_ctx, npts, n_atoms, radius, conformers):
    from autogrid_b200 import Diff
    _, prob = make_case(tmp_path, "elin", n_atoms, npts, seed=sum(npts) + n_atoms, radius=radius, ligand_types=["C"],
                        dsolvmap=False)
    e = prob.scalars["elec_map"]
    rng = np.random.default_rng(n_atoms)
    base = prob.arrays["coord"].reshape(-1, 3)
    coords = base + rng.normal(0.0, 0.2, (conformers,) + base.shape)
    coords[:, 0] = 0.0                       # on a grid point
    coords[:, 1] = [0.375, 0.1, -0.2]        # within 0.5 A of one
    w = np.zeros((conformers,) + prob.map_shape)
    w[:, e] = rng.normal(size=w[:, e].shape)
    shape = w.shape if conformers > 1 else prob.map_shape
    out = {}
    for prec in ("fp64", "fp32"):
        d = Diff(gpu_ctx, prob, prec, conformers=conformers)
        for k in range(conformers):
            d.set_atoms(coords[k], conformer=k)
        d.forward()
        g = d.backward(w.reshape(shape).astype(d.dtype))
        out[prec] = d.maps().reshape(w.shape)[:, e].astype(np.float64), g["coord"], g["charge"]
        d.close()
    ax = [(np.arange(n) - (n - 1) // 2) * prob.scalars["spacing"] for n in prob.n1]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    for k in range(conformers):
        size = np.zeros(x.shape)
        for c, q in zip(coords[k], prob.arrays["charge"]):
            r = np.sqrt((c[0] - x) ** 2 + (c[1] - y) ** 2 + (c[2] - z) ** 2)
            T = prob.arrays["r_epsilon_fn"][np.minimum((r * 128).astype(int), 8191)] * prob.scalars["coeff_estat"]
            size += np.abs(q) * T / np.maximum(r, 0.5)
        assert (np.abs(out["fp32"][0][k] - out["fp64"][0][k]) <= 265 * 2.0 ** -24 * size).all()
    off_grid = np.arange(prob.n_atoms) > 0
    for a, b in ((out["fp32"][1][..., off_grid, :], out["fp64"][1][..., off_grid, :]), (out["fp32"][2], out["fp64"][2])):
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)


@pytest.mark.parametrize("npts", [(2, 2, 2), (6, 6, 4), (16, 10, 8)])
@pytest.mark.parametrize("n_atoms,conformers", [(20, 1), (257, 2), (1030, 1)])
def test_fp64_e_map_and_adjoint(tmp_path, gpu_ctx, npts, n_atoms, conformers):
    """The FP64 twin, whose blocks hold 256 points (atoms) and share each sum
    out among 4 threads and tiles of 1,024, against numpy: fewer points or
    atoms than a block, remainders, more than one tile.  Each sum has at most
    2,000 terms, each within 1e-13 of itself (a few ulp of r move x = 128 r by
    1e-12 of a bin, whose step is below a tenth of its value): 1e-11 of the sum
    of the magnitudes bounds both.  The slope's division by the bin and by r
    takes two more digits."""
    from autogrid_b200 import Diff
    _, prob = make_case(tmp_path, "elin64", n_atoms, npts, seed=sum(npts) + n_atoms, ligand_types=["C"], dsolvmap=False)
    e, s = prob.scalars["elec_map"], prob.scalars
    rng = np.random.default_rng(n_atoms)
    base = prob.arrays["coord"].reshape(-1, 3)
    coords = base + rng.normal(0.0, 0.2, (conformers,) + base.shape)
    w = np.zeros((conformers,) + prob.map_shape)
    w[:, e] = rng.normal(size=w[:, e].shape)
    d = Diff(gpu_ctx, prob, "fp64", conformers=conformers)
    for k in range(conformers):
        d.set_atoms(coords[k], conformer=k)
    d.forward()
    g = d.backward(w.reshape(w.shape if conformers > 1 else prob.map_shape))
    got = d.maps().reshape(w.shape)[:, e]
    g_coord, g_q = g["coord"].reshape(conformers, -1, 3), g["charge"].reshape(conformers, -1)
    d.close()
    ax = [(np.arange(n) - (n - 1) // 2) * s["spacing"] for n in prob.n1]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    pts = np.stack([x, y, z], -1).reshape(-1, 3)
    T = prob.arrays["r_epsilon_fn"][:8192] * s["coeff_estat"]
    step = np.append(np.diff(T), 0.0)
    q = prob.arrays["charge"]
    for k in range(conformers):
        ref, size = np.zeros(len(pts)), np.zeros(len(pts))
        wk = w[k, e].ravel()
        for a in range(n_atoms):
            v = coords[k, a] - pts
            r = np.sqrt((v ** 2).sum(1))
            b = np.minimum((r * 128).astype(int), 8191)
            t, dt = T[b] + (r * 128 - b) * step[b], 128 * step[b]
            F = t / np.maximum(r, 0.5)
            dF = np.where(r > 0.5, dt / r - t / r ** 2, 2 * dt)
            ref += q[a] * F
            size += np.abs(q[a] * F)
            assert abs(g_q[k, a] - wk @ F) <= 1e-11 * (np.abs(wk) @ np.abs(F))
            c = (wk * q[a] * dF / r) @ v
            assert (np.abs(g_coord[k, a] - c) <= 1e-9 * np.abs((wk * q[a] * dF / r)[:, None] * v).sum(0) + 1e-30).all()
        assert (np.abs(got[k].ravel() - ref) <= 1e-11 * size).all()
