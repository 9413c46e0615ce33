"""Device memory and untuned choices of batches."""
import pytest

from conftest import make_case, tolerance_ok

pytestmark = pytest.mark.gpu


def test_large_ensemble_keeps_sums_of_few_chunks(tmp_path):
    """64 boxes of 3,000 atoms and 81^3 points make 157 waves of far units of
    2,048 atoms: the batch has room for no finer ones (of 512 atoms it would
    take 0.8 GB more)."""
    from autogrid_b200 import Batch, Context
    _, prob = make_case(tmp_path, "large", 3000, (80, 80, 80), seed=1, ligand_types=["C"], dielectric=40.0)
    ctx = Context(0)
    b = Batch(ctx, [prob] * 64)
    b.run()
    got = b.download(63)
    b.close()
    kept = ctx.cached_bytes()
    single = ctx.compute(prob)
    ctx.close()
    box = prob.points * 4
    # maps, the sums of two chunks, 1 MB of tables and atoms per box, and one block
    # of the cache
    assert tolerance_ok(got, single).all()
    assert kept <= 64 * (prob.n_maps * box + 2 * box + (1 << 20)) + (1 << 28)
