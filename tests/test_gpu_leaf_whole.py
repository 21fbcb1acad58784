"""init_knn's leaves as whole tiles in shared memory against the 128-row-tile
form and the FP32 form: same ids, same distance bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# leaves around a tile's edge and at the limits (2 rows, 512 and past it, where
# the general form takes over), few leaves (row blocks over several CTAs), exact
# rows (no error bound) and others, padded tails, the longest rows that fit (208
# dimensions, 4 tiles) and the first that do not, both metrics
@pytest.mark.parametrize("n,d,leaf,metric,kind", [
    (6000, 128, 500, "l2", "int"),
    (6000, 128, 128, "l2", "int"),
    (5003, 37, 129, "l2", "unit"),
    (4000, 16, 512, "ip", "int"),
    (4000, 100, 257, "ip", "unit"),
    (3000, 208, 512, "l2", "unit"),
    (3000, 209, 512, "l2", "int"),
    (2500, 48, 700, "l2", "mixed"),
    (3000, 130, 384, "l2", "int"),
    (3000, 20, 300, "l2", "mixed"),
    (2000, 8, 12, "l2", "int"),
])
def test_whole_leaves_equal_tiles(n, d, leaf, metric, kind, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    if kind == "int":
        x = rng.integers(0, 256, (n, d)) if d > 16 else rng.integers(-3, 4, (n, d))
    else:
        x = rng.standard_normal((n, d))
        x /= np.linalg.norm(x, axis=1, keepdims=True)
        if kind == "mixed":
            x[::2] = np.rint(8 * x[::2])
    x = np.ascontiguousarray(x, np.float32)
    K = min(100, leaf)
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, k=K, ef=2 * K, trees=6, leaf=leaf, metric=metric)
        fp32 = pipeline.aknn_build(ctx, x, k=K, ef=2 * K, trees=6, leaf=leaf, metric=metric, precision="fp32")
        monkeypatch.setenv("ANQI_B200_LEAF_WHOLE", "0")
        want = pipeline.aknn_build(ctx, x, k=K, ef=2 * K, trees=6, leaf=leaf, metric=metric)
    for other in (want, fp32):
        assert np.array_equal(got[0], other[0])
        assert np.array_equal(got[1].view(np.uint32), other[1].view(np.uint32))
