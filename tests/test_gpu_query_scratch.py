"""Device memory a small batch's search holds: one candidate list a query, and no
visited bitmaps or logs (the block-per-query form keeps its bitmap on the SM)."""
import numpy as np
import pytest

from test_zz_no_alloc import small_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 333])
def test_block_search_scratch(nq, monkeypatch):
    from anqi._lib import Context

    base, query, lifted, links, deg, tree, sc, m2, thr = small_index(n=5000, d=32, nq=333)
    query = np.ascontiguousarray(query[:nq])
    with Context(0) as ctx:
        ctx.index_load(base, lifted, deg, links, tree, sc, m2)
        ctx.set_thresholds(10, thr)
        before = ctx.device_bytes
        got = ctx.rknn_query(query, 10, 64)
        held = ctx.device_bytes - before
        # then the warp form, whose bitmaps come only now, and the block form again
        monkeypatch.setenv("ANQI_B200_BLOCK", "0")
        want = ctx.rknn_query(query, 10, 64)
        monkeypatch.delenv("ANQI_B200_BLOCK")
        again = ctx.rknn_query(query, 10, 64)
    for r in (got, again):
        assert np.array_equal(r.pred_off, want.pred_off) and np.array_equal(r.pred_ids, want.pred_ids)
        assert np.array_equal(r.n_dist, want.n_dist)
    # lists, results (128 a query, at least 1,024, twice) and the batch's own arrays
    lists, results = nq * len(base) * 4, 2 * max(1024, 128 * nq) * 4
    assert held <= lists + results + 1024 * nq + (1 << 20)
