"""The AKNN gather on component tables (csrc/component.cu) against the general
gather it stands in for: same ids and same distance bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clusters(sizes, d, integer, dup, seed):
    """Well separated clusters of the given sizes, rows shuffled together;
    `dup` repeats rows so that distances tie."""
    rng = np.random.default_rng(seed)
    parts = []
    for c, s in enumerate(sizes):
        center = np.zeros(d)
        center[c % d] = 4000.0 * (1 + c // d)
        x = rng.normal(0.0, 12.0, size=(s, d)) + center
        if dup:
            x = x[rng.integers(0, max(1, s // dup), size=s)]
        parts.append(np.rint(x) if integer else x)
    x = np.concatenate(parts).astype(np.float32)
    return x[rng.permutation(len(x))]


# word and register-instance edges (32, 33, 256 / 257, 640 / 641, 1152 / 1153,
# 2048 rows and one past it), dimensions with every kind of tail and past one
# staged block, ties, ef below the component size and below K + 1
@pytest.mark.parametrize("sizes,d,K,ef,integer,dup", [
    ([33, 32, 34, 64, 96], 16, 20, 600, False, 0),
    ([256, 257, 255], 128, 100, 600, True, 0),
    ([640, 641], 37, 100, 600, False, 0),
    ([1152, 1153], 130, 100, 600, False, 0),
    ([2048, 2049], 20, 100, 600, False, 0),
    ([300, 700], 5, 100, 600, True, 3),
    ([400, 500], 144, 64, 100, False, 0),
    ([400, 900], 24, 100, 40, True, 2),
    ([700, 300], 300, 200, 150, False, 0),
])
def test_component_gather_equals_general(sizes, d, K, ef, integer, dup, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    x = clusters(sizes, d, integer, dup, seed=sum(sizes) + d)
    with Context(0) as ctx:
        got = pipeline.aknn_build(ctx, x, k=K, ef=ef, trees=16, leaf=max(K + 20, 150))
        monkeypatch.setenv("ANQI_B200_GATHER_COMPONENTS", "0")
        want = pipeline.aknn_build(ctx, x, k=K, ef=ef, trees=16, leaf=max(K + 20, 150))
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    assert got[2]["pool_total"] == want[2]["pool_total"]
