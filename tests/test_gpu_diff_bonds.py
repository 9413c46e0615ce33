"""Gradients with respect to the bond vectors in FP32: the values that the
adjoint of the short-range maps sums for H-bond classes alone (position, charge,
rvector and rvector2 in one pass, and the closest hydrogen's rvector per point),
in every instantiation, against the FP64 twin.
"""
import numpy as np
import pytest

from conftest import make_case
from test_gpu_diff_rows import SETS

pytestmark = pytest.mark.gpu

ANGULAR = [n for n in SETS if n not in ("plain_small", "plain_16", "vina")]


@pytest.mark.parametrize("npts", [(8, 6, 4), (18, 10, 14)])
@pytest.mark.parametrize("name", ANGULAR)
def test_bond_vector_gradients(tmp_path, gpu_ctx, name, npts):
    """1e-3 of a norm, as for the coordinates: an FP32 distance takes the
    neighbouring bin in one pair of a thousand.  Per atom, of the largest
    gradient: a few of an atom's pairs at the most are such pairs, and what a
    bin's neighbour adds stays below a tenth of the pair."""
    from autogrid_b200 import Diff
    _, prob = make_case(tmp_path, name, 350, npts, seed=sum(npts), radius=10.0, **SETS[name])
    w = np.random.default_rng(1).normal(size=prob.map_shape)
    grads = {}
    for precision, dtype in (("fp64", np.float64), ("fp32", np.float32)):
        d = Diff(gpu_ctx, prob, precision)
        d.forward()
        grads[precision] = d.backward(w.astype(dtype))
        d.close()
    for key in ("rvector", "rvector2"):
        got, ref = grads["fp32"][key], grads["fp64"][key]
        scale = np.abs(ref).max()
        assert scale > 0.0 or (key == "rvector2" and name == "no_dsolv")  # no map of a donor probe: no A2 factor
        np.testing.assert_array_equal(got[(ref == 0).all(-1)], 0.0)
        assert np.linalg.norm(got - ref) <= 1e-3 * np.linalg.norm(ref), key
        assert np.abs(got - ref).max() <= 1e-2 * scale, key
