"""Tables with values that are not finite: the C ABI takes them, and the FP32
kernels do with them what the FP64 twins do.  H-bond min/max maps keep a NaN
that every pair of a class gives.
"""
import numpy as np
import pytest

from conftest import make_case, tolerance_ok

pytestmark = pytest.mark.gpu

LIGANDS = ["C", "HD", "NA", "OA"]


def tables_of(prob):
    """e_vdw_hb as [receptor type][map][bin] (a view)."""
    t, m = max(prob.scalars["n_rec_types"], 1), prob.scalars["n_atom_maps"]
    return prob.arrays["e_vdw_hb"][: t * m * 1024].reshape(t, m, 1024)


def types_of_class(prob, classes):
    return np.unique(prob.arrays["rec_type"][np.isin(prob.arrays["hbond"], classes)])


@pytest.mark.parametrize("npts,seed", [((30, 6, 8), 1), ((18, 18, 16), 2)])
@pytest.mark.parametrize("ligand,classes", [("HD", (4, 5)), ("NA", (1, 2))])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_minmax_maps_keep_what_is_not_finite(tmp_path, gpu_ctx, ligand, classes, value, npts, seed):
    """Every pair of the classes that enter a map's H-bond min/max has the value."""
    _, prob = make_case(tmp_path, "minmax", 25, npts, seed=seed, spacing=1.3, ligand_types=LIGANDS)
    finite = gpu_ctx.compute(prob, "fp32").reshape(prob.n_maps, -1)
    m = LIGANDS.index(ligand)
    tables_of(prob)[types_of_class(prob, classes), m] = value
    twin = gpu_ctx.compute(prob, "fp64").reshape(prob.n_maps, -1)
    hit = ~np.isfinite(twin[m])
    assert hit.any() and not hit.all() and np.isfinite(np.delete(twin, m, 0)).all()
    plan = gpu_ctx.plan(prob)
    plan.run()
    planned = plan.download()
    plan.close()
    for got in (gpu_ctx.compute(prob, "fp32"), planned):
        got = got.reshape(prob.n_maps, -1)
        np.testing.assert_array_equal(got[m][hit], twin[m][hit].astype(np.float32))
        assert tolerance_ok(got[m][~hit], twin[m][~hit]).all()
        np.testing.assert_array_equal(np.delete(got, m, 0), np.delete(finite, m, 0))


def test_gradient_with_a_dielectric_beyond_every_pair(tmp_path, gpu_ctx):
    """Dielectric values at distances that no atom and point have do not reach
    the gradient (the kernels pad the box to whole frames)."""
    from autogrid_b200 import Diff
    _, prob = make_case(tmp_path, "far_eps", 200, (4, 6, 2), seed=3, ligand_types=["C", "OA"])
    n1, ne, sp = prob.n1, prob.ne, prob.scalars["spacing"]
    c = prob.arrays["coord"].reshape(-1, 3)
    lo, hi = -np.array(ne) * sp, (np.array(n1) - 1 - np.array(ne)) * sp
    reach = np.sqrt((np.maximum(abs(c - lo), abs(c - hi)) ** 2).sum(1).max())
    w = np.zeros(prob.map_shape, np.float32)
    w[prob.scalars["elec_map"]] = np.random.default_rng(1).normal(size=prob.map_shape[1:])
    assert prob.scalars["dddiel"]
    grads = []
    for value in (None, np.nan, np.inf):
        if value is not None:
            prob.arrays["r_epsilon_fn"][int(reach * 128) + 4:] = value
        d = Diff(gpu_ctx, prob, "fp32")
        d.forward()
        grads.append((d.maps(), d.backward(w)))
        d.close()
    for maps, g in grads[1:]:
        np.testing.assert_array_equal(maps, grads[0][0])
        for key in ("coord", "charge"):
            norm = np.linalg.norm(grads[0][1][key])
            assert np.linalg.norm(g[key] - grads[0][1][key]) <= 1e-6 * norm, key
