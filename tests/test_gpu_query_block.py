"""The block-per-query search of small batches against the warp-per-query
search: same candidates in the same order, same results, same counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(n, d, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "unit":
        x = rng.standard_normal((n, d))
        return (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)
    c = rng.uniform(0, 128, size=(max(4, n // 60), d))
    x = np.rint(np.clip(c[rng.integers(0, len(c), n)] + rng.normal(0, 20, (n, d)), 0, 255)).astype(np.float32)
    return x[rng.integers(0, n // 2, n)] if kind == "dup" else x


# the compile-time dimension (128) and the general one with every tail, beams
# from one entry to more than a block's threads, one query to more than one per
# SM, tied distances, the ip metric's per-query radius
@pytest.mark.parametrize("n,d,kind,metric,nq,k,L", [
    (3000, 128, "mixture", "l2", 1, 10, 128),
    (3000, 128, "dup", "l2", 97, 50, 257),
    (5000, 128, "unit", "ip", 160, 100, 33),
    (2500, 100, "unit", "ip", 333, 0, 0),
    (2500, 37, "dup", "l2", 64, 100, 600),
    (1500, 8, "mixture", "l2", 31, 10, 1),
    (2000, 250, "unit", "l2", 5, 50, 1024),
])
def test_block_search_equals_warp_search(n, d, kind, metric, nq, k, L, monkeypatch):
    from anqi import lrq_fit, pipeline
    from anqi._lib import Context

    x = rows(n + nq, d, kind, n + d)
    base, query = np.ascontiguousarray(x[:n]), np.ascontiguousarray(x[n:])
    rng = np.random.default_rng(nq)
    ks = k or rng.choice(np.array([10, 50, 100], np.uint32), nq)
    Ls = L or rng.integers(4, 300, nq).astype(np.uint32)
    with Context(0) as ctx:
        ids, keys, _ = pipeline.aknn_build(ctx, base, metric=metric)
        f = [np.asarray(a, np.float32) for a in lrq_fit.train_gpu(keys, n, log=lambda s: None)]
        coeff, codes = ctx.lrq_encode(keys, *f)
        lifted, m2, sc = ctx.lift(base, keys[:, -1], metric=metric)
        deg, links, tree, _ = pipeline.graph_build(ctx, lifted, ids)
        ctx.index_load(base, lifted, deg, links, tree, sc, m2, metric=metric)
        ctx.verifier_load_bits(coeff, codes.reshape(-1), None, 100, *f, 8, signed_keys=metric == "ip")
        for kk in (10, 50, 100):
            ctx.verifier_materialize(kk)
        monkeypatch.setenv("ANQI_B200_BLOCK", "0")
        want = ctx.rknn_query(query, ks, Ls, keep_candidates=True)
        monkeypatch.delenv("ANQI_B200_BLOCK")
        got = ctx.rknn_query(query, ks, Ls, keep_candidates=True)
        assert want.stats["warps_per_block"] * want.stats["candidate_tile"] and got.stats["visited_table"] == 0
        ctx.query_upload(query, ks, Ls)
        for _ in range(2):  # the second replays the captured graph
            ctx.query_run_graph(True)
        graph = ctx.query_download(with_candidates=True)
    for r in (got, graph):
        assert np.array_equal(r.n_dist, want.n_dist)
        assert np.array_equal(r.cand_off, want.cand_off) and np.array_equal(r.cand_ids, want.cand_ids)
        assert np.array_equal(r.pred_off, want.pred_off) and np.array_equal(r.pred_ids, want.pred_ids)
    assert want.n_dist.min() > 0
