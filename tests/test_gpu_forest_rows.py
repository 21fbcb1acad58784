"""The forest's sides from the rows' bf16 copies against those from the rows: the
same trees, so the same lists out of two trees' leaves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# padded tails (a K group short, an odd pair of them, the K-chunked row length),
# rows whose rounding decides nothing (integers), some (unit rows) and most sides
# (lengths over six decades), duplicates (margins of zero, hashed sides), chunks
# past one and short last ones
@pytest.mark.parametrize("n,d,metric,kind", [
    (9000, 128, "l2", "int"),
    (7001, 37, "l2", "unit"),
    (5000, 100, "ip", "unit"),
    (6000, 24, "l2", "long"),
    (4100, 8, "ip", "long"),
    (5000, 16, "l2", "dup"),
    (3000, 300, "l2", "unit"),
    (3000, 3, "l2", "offset"),
])
def test_sides_from_bf16_rows(n, d, metric, kind, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d))
    if kind == "int":
        x = np.rint(40 * x)
    elif kind == "long":
        x *= 10.0 ** rng.uniform(-3, 3, (n, 1))
    elif kind == "offset":
        x += 1000.0
    else:
        x /= np.linalg.norm(x, axis=1, keepdims=True)
        if kind == "dup":
            x = x[rng.integers(0, n // 20, n)]
    x = np.ascontiguousarray(x, np.float32)
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, k=20, ef=20, trees=2, leaf=50, metric=metric)
        monkeypatch.setenv("ANQI_B200_FOREST_BF16", "0")
        want = pipeline.aknn_build(ctx, x, k=20, ef=20, trees=2, leaf=50, metric=metric)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
