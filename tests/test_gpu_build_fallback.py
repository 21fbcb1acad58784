"""Builds whose optional device buffers cannot be had (ANQI_FAULT_OPTIONAL_ALLOC):
the forms that need less memory take over, with the same output."""
import numpy as np
import pytest

from test_gpu_component import clusters

pytestmark = pytest.mark.gpu

OPTIONAL_ALLOC = 2


def same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1].view(np.uint32), b[1].view(np.uint32))


def test_graph_without_component_tables():
    from anqi import pipeline
    from anqi._lib import Context

    x = clusters([500, 400, 300], 30, False, 0, seed=4)
    with Context(0) as ctx:
        ids, keys, _ = pipeline.aknn_build(ctx, x, k=100, trees=16, leaf=150)
        lifted = ctx.lift(x, keys[:, -1])[0]
        want = pipeline.graph_build(ctx, lifted, ids)
        ctx.inject_fault(OPTIONAL_ALLOC)
        got = pipeline.graph_build(ctx, lifted, ids)
        ctx.inject_fault(0)
        again = pipeline.graph_build(ctx, lifted, ids)
    for g in (got, again):
        assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1])
        assert g[3]["pool_total"] == want[3]["pool_total"]


@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_source_without_optional_buffers(metric):
    from anqi import pipeline
    from anqi._lib import Context

    x = clusters([500, 400, 300, 3000], 30, False, 0, seed=5)
    opts = dict(k=50, trees=16, leaf=150, metric=metric)
    with Context(0) as ctx:
        want = pipeline.aknn_build(ctx, x, **opts)
        ctx.inject_fault(OPTIONAL_ALLOC)
        got = pipeline.aknn_build(ctx, x, **opts)
        ctx.inject_fault(0)
        again = pipeline.aknn_build(ctx, x, **opts)
    assert same(got, want) and same(again, want)
    assert got[2]["pool_total"] == want[2]["pool_total"]
