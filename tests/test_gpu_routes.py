"""Which kernels a call runs: each switch's two arms, which other tests compare by
their results, do take different forms."""
import re

import numpy as np
import pytest

from test_gpu_component import clusters
from test_zz_no_alloc import small_index

pytestmark = pytest.mark.gpu


def kernels(run):
    """Names of the library's kernels that run() launches."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
    return {m.group(1) for e in p.key_averages() if (m := re.search(r"anqi::.*?(\w+_kernel)\b", e.key))}


def unit(n, d, seed):
    x = np.random.default_rng(seed).standard_normal((n, d)).astype(np.float32)
    return x / np.linalg.norm(x, axis=1, keepdims=True)


@pytest.mark.parametrize("d", [32, 128])
def test_query_forms(d, monkeypatch):
    from anqi._lib import Context

    base, query, lifted, links, deg, tree, sc, m2, thr = small_index(n=2000, d=d, nq=60)
    with Context(0) as ctx:
        ctx.index_load(base, lifted, deg, links, tree, sc, m2)
        ctx.set_thresholds(10, thr)
        few = kernels(lambda: ctx.rknn_query(query, 10, 64))
        many = kernels(lambda: ctx.rknn_query(np.tile(query, (100, 1)), 10, 64))
        monkeypatch.setenv("ANQI_B200_BLOCK", "0")
        off = kernels(lambda: ctx.rknn_query(query, 10, 64))
    assert "rknn_search_block_kernel" in few and "rknn_search_kernel" not in few
    for k in (many, off):
        assert "rknn_search_kernel" in k and "rknn_search_block_kernel" not in k


@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_gather_forms(metric, monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    x = unit(3000, 24, 1)
    opts = dict(k=50, ef=100, trees=4, leaf=100, metric=metric)
    with Context(0) as ctx:
        block = kernels(lambda: pipeline.aknn_build(ctx, x, **opts))
        monkeypatch.setenv("ANQI_B200_GATHER_BLOCK", "0")
        warp = kernels(lambda: pipeline.aknn_build(ctx, x, **opts))
    assert "gather_block_kernel" in block and "gather_kernel" not in block
    assert "gather_kernel" in warp and "gather_block_kernel" not in warp


def test_component_forms(monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    x = clusters([300, 200, 400], 20, False, 0, seed=1)
    with Context(0) as ctx:
        run = lambda: pipeline.aknn_build(ctx, x, k=100, trees=8, leaf=150)  # noqa: E731
        ids, keys, _ = run()
        lifted = ctx.lift(x, keys[:, -1])[0]
        graph = lambda: pipeline.graph_build(ctx, lifted, ids)  # noqa: E731
        source, built = kernels(run), kernels(graph)
        monkeypatch.setenv("ANQI_B200_GATHER_COMPONENTS", "0")
        monkeypatch.setenv("ANQI_B200_GRAPH_COMPONENTS", "0")
        source_off, built_off = kernels(run), kernels(graph)
        monkeypatch.delenv("ANQI_B200_GATHER_COMPONENTS")
        monkeypatch.delenv("ANQI_B200_GRAPH_COMPONENTS")
        ctx.inject_fault(2)  # no memory for the optional forms
        source_full, built_full = kernels(run), kernels(graph)
    assert "comp_search_kernel" in source and not source & {"gather_kernel", "gather_block_kernel"}
    assert {"comp_select_kernel", "comp_commit_kernel"} <= built and "gather_kernel" not in built
    assert "forest_sides_bf16_kernel" in source
    for k in (source_off, source_full):
        assert "comp_search_kernel" not in k and "gather_block_kernel" in k
    for k in (built_off, built_full):
        assert "comp_select_kernel" not in k and "gather_kernel" in k
    assert "forest_sides_kernel" in source_full and "forest_sides_bf16_kernel" not in source_full


def test_leaf_and_side_forms(monkeypatch):
    from anqi import pipeline
    from anqi._lib import Context

    x = unit(2000, 40, 2)
    opts = dict(k=20, ef=40, trees=2, leaf=100)
    with Context(0) as ctx:
        whole = kernels(lambda: pipeline.aknn_build(ctx, x, **opts))
        longer = kernels(lambda: pipeline.aknn_build(ctx, x, k=20, ef=40, trees=2, leaf=700))
        monkeypatch.setenv("ANQI_B200_LEAF_WHOLE", "0")
        monkeypatch.setenv("ANQI_B200_FOREST_BF16", "0")
        off = kernels(lambda: pipeline.aknn_build(ctx, x, **opts))
    assert {"tc_leaf_kernel", "forest_sides_bf16_kernel"} <= whole and "tc_filter_kernel" not in whole
    assert "tc_filter_kernel" in longer and "tc_leaf_kernel" not in longer
    assert {"tc_filter_kernel", "forest_sides_kernel"} <= off
    assert not off & {"tc_leaf_kernel", "forest_sides_bf16_kernel"}
