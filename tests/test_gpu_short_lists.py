"""init_knn lists that stay shorter than K (small leaves, few trees): the FP32 form
leaves the rest of a list empty, so its output is the BF16 form's, every time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,leaf,trees,metric", [
    (3000, 24, 50, 1, "l2"), (3000, 128, 30, 2, "l2"), (2000, 37, 60, 1, "ip"),
])
def test_short_lists(n, d, leaf, trees, metric):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    with Context(0) as ctx:
        want = pipeline.aknn_build(ctx, x, k=100, ef=20, leaf=leaf, trees=trees, metric=metric)
        for _ in range(2):
            got = pipeline.aknn_build(ctx, x, k=100, ef=20, leaf=leaf, trees=trees, metric=metric, precision="fp32")
            assert np.array_equal(got[0], want[0])
            assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


def test_short_lists_stage():
    from anqi._lib import Context

    rng = np.random.default_rng(5)
    x = rng.standard_normal((90, 16)).astype(np.float32)
    off, leaves = np.array([0, 30, 60, 90], np.uint64), rng.permutation(90).astype(np.uint32)
    ids, dist = np.empty((90, 50), np.uint32), np.empty((90, 50), np.float32)
    with Context(0) as ctx:
        ctx._check(ctx.lib.anqi_aknn_init(ctx.h, x, 90, 16, off, leaves, 3, 50, ids, dist), "aknn_init")
    assert (ids[:, :29] < 90).all()
    assert (ids[:, 29:] == 0xFFFFFFFF).all() and (dist[:, 29:] == np.finfo(np.float32).max).all()
