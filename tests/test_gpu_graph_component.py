"""Select and commit of the graph build on component tables against the
general gather and commit: same degrees and links."""
import numpy as np
import pytest

from test_gpu_component import clusters

pytestmark = pytest.mark.gpu


# register-instance edges, an explore range that ends searches early and one
# that exhausts them, the pool cap below and above the component size, ties,
# every degree bound, and one component too large (the general path throughout)
@pytest.mark.parametrize("sizes,d,degree,explore,ef_alpha,integer,dup", [
    ([120, 150, 256, 257], 30, 48, 100, 8, False, 0),
    ([640, 641, 1152, 1153], 16, 48, 100, 8, False, 0),
    ([2048, 300], 126, 48, 100, 8, False, 0),
    ([500, 400], 10, 16, 20, 4, True, 3),
    ([500, 400], 10, 64, 30, 64, True, 4),
    ([200, 200], 12, 1, 10, 1, False, 0),
    ([2049, 300], 8, 48, 100, 8, False, 0),
])
def test_component_graph_equals_general(sizes, d, degree, explore, ef_alpha, integer, dup, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    x = clusters(sizes, d, integer, dup, seed=sum(sizes) + d)
    with Context(0) as ctx:
        ids, keys, _ = pipeline.aknn_build(ctx, x, k=100, trees=16, leaf=150)
        lifted = ctx.lift(x, keys[:, -1])[0]
        opts = dict(degree=degree, explore=explore, ef_alpha=ef_alpha)
        deg, links, _, st = pipeline.graph_build(ctx, lifted, ids, **opts)
        monkeypatch.setenv("ANQI_B200_GRAPH_COMPONENTS", "0")
        wdeg, wlinks, _, wst = pipeline.graph_build(ctx, lifted, ids, **opts)
    assert np.array_equal(deg, wdeg) and np.array_equal(links, wlinks)
    assert st["pool_total"] == wst["pool_total"] and deg.max() <= degree
