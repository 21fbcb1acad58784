"""Queries that hold NaN or infinities, or overflow, in every form of the search:
they find nothing, and the batch's other queries find what they do without them."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import DeviceIndex, bind, device_rows, device_u32, padded, small_index

pytestmark = pytest.mark.gpu


def spoil(query, seed):
    """The batch with every fifth query made non-finite, and which ones are."""
    rng = np.random.default_rng(seed)
    q, bad = query.copy(), np.zeros(len(query), bool)
    bad[::5] = True
    for t, i in enumerate(np.flatnonzero(bad)):
        j = rng.integers(0, q.shape[1])
        if t % 4 == 0:
            q[i, j] = np.nan
        elif t % 4 == 1:
            q[i] = np.nan
        elif t % 4 == 2:
            q[i, j] = np.inf
        else:
            q[i] = 3e38
    return q, bad


# d + 2 with the compile-time distance loops (d = 128) and without; beams of one
# entry, below and past what one expansion brings; the block form (the default for
# so few), the warp form and the captured graph
@pytest.mark.parametrize("d,L", [(128, 1), (128, 40), (128, 300), (20, 64)])
def test_nonfinite_queries_find_nothing(d, L, monkeypatch):
    from anqi._lib import Context

    base, query, lifted, links, deg, tree, sc, m2, thr = small_index(n=3000, d=d, nq=100)
    spoiled, bad = spoil(query, d)
    with Context(0) as ctx:
        ctx.index_load(base, lifted, deg, links, tree, sc, m2)
        ctx.set_thresholds(10, thr)
        for block in ("1", "0"):
            monkeypatch.setenv("ANQI_B200_BLOCK", block)
            want = ctx.rknn_query(query, 10, L)
            got = [ctx.rknn_query(spoiled, 10, L)]
            ctx.query_upload(spoiled, 10, L)
            for _ in range(2):  # the second replays the captured graph
                ctx.query_run_graph(False)
            got.append(ctx.query_download())
            for r in got:
                for i in range(len(query)):
                    if bad[i]:
                        assert len(r.pred(i)) == 0
                    else:
                        assert np.array_equal(r.pred(i), want.pred(i)) and r.n_dist[i] == want.n_dist[i]


def test_nonfinite_queries_without_allocation():
    import torch

    from anqi._lib import ANQI_OK, Context, load_library

    d, L, cap = 32, 64, 512
    base, query, lifted, links, deg, tree, sc, m2, thr = small_index(d=d, nq=100)
    spoiled, bad = spoil(query, d)
    with Context(0) as ctx:
        ctx.index_load(base, lifted, deg, links, tree, sc, m2)
        ctx.set_thresholds(10, thr)
        want = ctx.rknn_query(query, 10, L)
    lib = bind(load_library())
    n, bs, ls = len(base), d, (d + 2 + 3) // 4 * 4
    t = [device_rows(torch, base, bs, n), device_rows(torch, lifted, ls, n), device_u32(torch, deg),
         device_u32(torch, links), device_u32(torch, tree.left), device_u32(torch, tree.right),
         torch.from_numpy(tree.offset.copy()).cuda(), padded(torch, tree.hyperplane, ls),
         device_u32(torch, tree.leaf_first()), device_rows(torch, thr[:, None], 1), padded(torch, spoiled, bs)]
    p = [a.data_ptr() for a in t]
    ix = DeviceIndex(n, d, links.shape[1], p[0], bs, p[1], ls, p[2], p[3], tree.n_nodes, p[4], p[5], p[6], p[7], p[8],
                     sc, m2)
    cnt, nd = (torch.zeros(len(query), dtype=torch.int32, device="cuda") for _ in range(2))
    ids = torch.full((len(query), cap), -1, dtype=torch.int32, device="cuda")
    rc = lib.anqi_rknn_query_noalloc(C.byref(ix), p[10], len(query), p[9], L, cap, cnt.data_ptr(), ids.data_ptr(),
                                     nd.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == ANQI_OK
    cnt, ids = cnt.cpu().numpy(), ids.cpu().numpy().view(np.uint32)
    for i in range(len(query)):
        assert np.array_equal(ids[i, :cnt[i]], [] if bad[i] else want.pred(i))
