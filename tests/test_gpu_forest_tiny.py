"""The forest's sides from bf16 rows where a hyperplane's squares underflow (it is
the difference of two tiny rows) and other rows are huge: the same lists as with
sides from the FP32 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,metric,tiny,huge", [(8, "l2", 1e-23, 1e18), (24, "l2", 3e-24, 5e17)])
def test_sides_of_tiny_hyperplanes(d, metric, tiny, huge, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(d)
    n = 60_000
    x = rng.standard_normal((n, d)) * np.where(rng.random((n, 1)) < 0.5, tiny, huge)
    x = np.ascontiguousarray(x, np.float32)
    opts = dict(k=20, ef=20, trees=2, leaf=50, metric=metric)
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, **opts)
        monkeypatch.setenv("ANQI_B200_FOREST_BF16", "0")
        want = pipeline.aknn_build(ctx, x, **opts)
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
