"""Far-field kernel units at the edges of their tiling: boxes whose last frame
holds 1-4 or more rows and columns, atom counts around the 32-atom blocks that
the two halves of a CTA share out, the clamped table and a constant dielectric.

The e map is compared with the FP64 oracle.  A point's sum is built from runs
of at most 256 terms, so rounding stays below 255 + 8 units of 2^-24 of the sum
of the terms' magnitudes (8: the terms' own roundings); a pair in a wrong table
bin is off by a thousandth of its term, more than that for the small counts.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu

BOXES = [(2, 2, 2), (8, 4, 6), (30, 8, 8), (32, 10, 2), (40, 14, 10), (56, 6, 16)]


def _bound(prob):
    a, s = prob.arrays, prob.scalars
    ax = [(np.arange(n) - (n - 1) // 2) * s["spacing"] for n in prob.n1]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    pts = np.stack([x, y, z], -1).reshape(-1, 3)
    c, q = a["coord"].reshape(-1, 3), a["charge"]
    out = np.zeros(len(pts))
    for i in range(len(q)):
        r = np.sqrt(((c[i] - pts) ** 2).sum(1))
        k = np.minimum((r * 128).astype(int), 8191)
        T = a["r_epsilon_fn"][k] if s["dddiel"] else s["invdielcal"]
        out += np.abs(q[i]) * T * s["coeff_estat"] / np.maximum(r, 0.5)
    return 263 * 2.0 ** -24 * out + 1e-30


@pytest.mark.parametrize("mode", ["table", "clamp", "const"])
@pytest.mark.parametrize("n_atoms", [40, 65, 513])
@pytest.mark.parametrize("npts", BOXES)
def test_e_map_against_oracle(tmp_path, gpu_ctx, npts, n_atoms, mode):
    from oracle.oracle import oracle_points
    kw = dict(radius=160.0) if mode == "clamp" else {}
    _, prob = make_case(tmp_path, "far", n_atoms, npts, seed=sum(npts) + n_atoms, ligand_types=["C"],
                        dielectric=40.0 if mode == "const" else -0.1465, **kw)
    e = prob.scalars["elec_map"]
    ref, flags = oracle_points(prob)
    got = gpu_ctx.compute(prob, "fp32").reshape(prob.n_maps, -1)[e]
    off = np.abs(got - ref[e]) > _bound(prob)
    assert not (off & (flags == 0)).any()
    plan = gpu_ctx.plan(prob)
    plan.run()
    again = plan.download().reshape(prob.n_maps, -1)[e]
    assert not ((np.abs(again - ref[e]) > _bound(prob)) & (flags == 0)).any()
    plan.close()


@pytest.mark.parametrize("n_atoms", [31, 97, 1030])
@pytest.mark.parametrize("npts", [(8, 2, 8), (34, 10, 10), (10, 4, 12), (4, 12, 18)])
def test_e_map_of_boxes_cut_in_z(tmp_path, gpu_ctx, npts, n_atoms):
    """Last z frames of 1, 3 and 5 planes, whose warps share the atoms out
    among 8, 4 and 2 groups: fewer blocks of 32 atoms than groups, a rest, and
    more than one tile."""
    from oracle.oracle import oracle_points
    _, prob = make_case(tmp_path, "cut", n_atoms, npts, seed=sum(npts) + n_atoms, ligand_types=["C"])
    e = prob.scalars["elec_map"]
    ref, flags = oracle_points(prob)
    got = gpu_ctx.compute(prob, "fp32").reshape(prob.n_maps, -1)[e]
    assert not ((np.abs(got - ref[e]) > _bound(prob)) & (flags == 0)).any()


@pytest.mark.parametrize("mode", ["table", "beyond_256A", "const"])
@pytest.mark.parametrize("npts,n_atoms", [((2, 2, 2), 3), ((14, 8, 6), 300), ((16, 6, 8), 257), ((34, 18, 4), 1100)])
def test_fp64_e_map(tmp_path, gpu_ctx, npts, n_atoms, mode):
    """The FP64 twin's bricks, atom chunks and fixed-point bins, against the
    nested hypot in numpy; points with a pair within 1e-9 bins of an edge are
    left out (the two hypots may differ there), and the rest agrees to the
    rounding of the sums."""
    kw = dict(radius=300.0) if mode == "beyond_256A" else {}
    _, prob = make_case(tmp_path, "far64", max(n_atoms, 20), npts, seed=sum(npts) + n_atoms, ligand_types=["C"],
                        dielectric=40.0 if mode == "const" else -0.1465, **kw)
    a, s = prob.arrays, prob.scalars
    ax = [(np.arange(n) - (n - 1) // 2) * s["spacing"] for n in prob.n1]
    z, y, x = (v.ravel() for v in np.meshgrid(ax[2], ax[1], ax[0], indexing="ij"))
    c, q = a["coord"].reshape(-1, 3), a["charge"]
    ref, size, tie = np.zeros(x.size), np.zeros(x.size), np.zeros(x.size, bool)
    for i in range(len(q)):
        r = np.maximum(np.hypot(c[i, 0] - x, np.hypot(c[i, 1] - y, c[i, 2] - z)), 1e-6)
        tie |= np.abs(r * 128 - np.rint(r * 128)) < 1e-9
        f = a["r_epsilon_fn"][np.minimum((r * 128).astype(int), 8191)] if s["dddiel"] else s["invdielcal"]
        term = q[i] / np.maximum(r, 0.5) * f * s["coeff_estat"]
        ref += term
        size += np.abs(term)
    got = gpu_ctx.compute(prob, "fp64").reshape(prob.n_maps, -1)[s["elec_map"]]
    free = ~tie if s["dddiel"] else slice(None)
    assert (np.abs(got - ref) <= 1e-12 * size + 1e-300)[free].all()
