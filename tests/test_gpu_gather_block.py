"""The block-per-row AKNN gather against the warp-per-row one: same ids and same
distance bits, on lists that form one large component."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# both metrics, dimensions with every kind of tail (ip: the last dim mod 8
# products are fused), chunked rows (128), ids past one chunk of threads (hubs at
# d = 8), K above a block's threads, an explore range below them and one the
# search exhausts, ties and duplicate rows
@pytest.mark.parametrize("n,d,metric,kind,K,ef", [
    (3000, 128, "l2", "unit", 100, 600),
    (2600, 37, "l2", "dup", 100, 600),
    (4000, 8, "l2", "int", 100, 300),
    (2500, 96, "ip", "unit", 100, 600),
    (2500, 99, "ip", "dup", 50, 120),
    (2600, 20, "ip", "int", 200, 400),
    (3000, 16, "l2", "unit", 150, 160),
])
def test_block_gather_equals_warp_gather(n, d, metric, kind, K, ef, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d))
    if kind == "int":
        x = np.rint(3 * x)
    else:
        x /= np.linalg.norm(x, axis=1, keepdims=True)
    if kind == "dup":
        x = x[rng.integers(0, n // 2, n)]
    x = np.ascontiguousarray(x, np.float32)
    monkeypatch.setenv("ANQI_B200_GATHER_COMPONENTS", "0")
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, k=K, ef=ef, trees=8, leaf=max(K + 20, 150), metric=metric)
        monkeypatch.setenv("ANQI_B200_GATHER_BLOCK", "0")
        want = pipeline.aknn_build(ctx, x, k=K, ef=ef, trees=8, leaf=max(K + 20, 150), metric=metric)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    assert got[2]["pool_total"] == want[2]["pool_total"]
