"""init_knn's whole leaves on signed integer rows whose l2 keys pass 2^24, where
the FP32 key is a rounded one and ties at the K-th key are many: same ids, same
distance bits as the 128-row-tile form and the FP32 form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# two clusters of opposite signs and entries +-{255, 256}: a list's tail crosses
# to the other one, with keys about 2^25; and the largest entries whose keys cannot
# pass 2^24 (4 * 128 * 181^2 = 16,773,632)
@pytest.mark.parametrize("n,d,K,leaf,first,big", [
    (400, 128, 150, 200, 120, 256),
    (300, 128, 100, 150, 60, 256),
    (500, 127, 200, 260, 180, 256),
    (400, 128, 150, 200, 120, 181),
])
def test_signed_leaves_equal_fp32(n, d, K, leaf, first, big, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    ones = rng.integers(d // 2, d // 2 + 2, (n, 1))
    x = np.where(np.argsort(rng.random((n, d)), axis=1) < ones, big, big - 1)
    x[rng.permutation(n)[first:]] *= -1
    x = np.ascontiguousarray(x, np.float32)
    # one expansion a row: what init_knn misses is mostly missed by the gather too
    opts = dict(k=K, ef=1, trees=24, leaf=leaf)
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, **opts)
        fp32 = pipeline.aknn_build(ctx, x, precision="fp32", **opts)
        monkeypatch.setenv("ANQI_B200_LEAF_WHOLE", "0")
        want = pipeline.aknn_build(ctx, x, **opts)
    assert got[1].max() > 2 ** 24 or big < 256
    for other in (want, fp32):
        assert np.array_equal(got[0], other[0])
        assert np.array_equal(got[1].view(np.uint32), other[1].view(np.uint32))
