"""The AKNN source over rows that hold NaN or infinities, or whose norms overflow:
the block-per-row gather's lists are the warp-per-row gather's, and every id is a
row's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# FP32 init_knn over leaves too small to fill a list, which so takes in rows at
# infinite distance; both metrics, the second also without component tables (their
# components are left to the general gather anyway, being non-finite)
@pytest.mark.parametrize("n,d,metric,components", [
    (2000, 24, "l2", "1"), (2000, 128, "l2", "0"), (1500, 37, "ip", "1"), (1500, 1030, "l2", "1"),
])
def test_block_gather_of_nonfinite_rows(n, d, metric, components, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    spoil = rng.permutation(n)[: n // 10]
    x[spoil[::4], 0] = np.nan
    x[spoil[1::4]] = np.nan
    x[spoil[2::4], d - 1] = np.inf
    x[spoil[3::4]] *= np.float32(1e25)
    monkeypatch.setenv("ANQI_B200_GATHER_COMPONENTS", components)
    opts = dict(k=100, ef=200, trees=2, leaf=60, metric=metric, precision="fp32")
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, **opts)
        monkeypatch.setenv("ANQI_B200_GATHER_BLOCK", "0")
        want = pipeline.aknn_build(ctx, x, **opts)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    ids = got[0][got[0] != 0xFFFFFFFF]
    assert ids.size and ids.max() < n
    assert np.isin(ids, spoil).any()  # rows at infinite distance did come into lists
