"""The work that programs have this library do, as cases that can be timed and
compared: reverse-kNN queries, the index build's stages, the exact ground
truth and the LRQ verifier's fit.

Kinds of case (``kind``) and what each stands for:

* ``query``: a batch of reverse-kNN queries against a resident index, from host
  vectors to host results.  ``call`` "host" is ``Context.rknn_query`` (with
  ``pinned`` as a serving loop holds its buffers), "graph" the resident form:
  upload, one CUDA-graph replay, download.  ``k`` / ``L`` 0 draw each query's k
  from {10, 50, 100} and its beam width from [64, 600].
* ``aknn``: the approximate top-100 source build (build_aknn_source).
* ``graph``: the G48 build over lifted rows from the AKNN lists (rknn_query's
  index build).
* ``truth``: dataset_gt: exact top-100 thresholds, bounded by the AKNN lists,
  then the exact reverse-kNN CSR at k = 10, 50 and 100.
* ``verifier``: the LRQ verifier from a cutoff matrix: fit, encode of every
  row, thresholds at k = 10, 50 and 100.
* ``objective``: one step of the LRQ gradient fit: objective and gradients.

Data: "mixture" rows are non-negative integers from a Gaussian mixture (the
shape of SIFT-like descriptors), "unit" rows L2-normalised N(0, 1) vectors
(embeddings).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "anqi-implementation_b200"))

KS = (10, 50, 100)


def listed():
    return [
        # an interactive lookup: one query, latency is all that counts
        dict(name="query_one", kind="query", n=50_000, d=128, data="mixture", metric="l2", nq=1, k=10, L=128,
             call="host", pinned=False),
        # a small odd batch over embeddings under the ip metric, candidates kept for an evaluation
        dict(name="query_ip", kind="query", n=60_000, d=100, data="unit", metric="ip", nq=333, k=50, L=85,
             call="host", pinned=False),
        # a stream of batches whose queries bring their own k and beam width
        dict(name="query_mixed", kind="query", n=200_000, d=128, data="mixture", metric="l2", nq=10_000, k=0, L=0,
             call="graph", pinned=False),
        # the headline batch: 10,000 queries at three k over a million rows
        dict(name="query_million", kind="query", n=1_000_000, d=128, data="mixture", metric="l2", nq=30_000, k=0,
             L=128, call="host", pinned=True),
        # long rows (GIST-like)
        dict(name="query_wide", kind="query", n=30_000, d=960, data="unit", metric="l2", nq=2_000, k=0, L=128,
             call="host", pinned=False),
        # a small ragged collection's source build
        dict(name="aknn_small", kind="aknn", n=5_003, d=37, data="unit", metric="l2"),
        # embeddings under the ip metric: angular forest, unclustered lists
        dict(name="aknn_ip", kind="aknn", n=100_000, d=100, data="unit", metric="ip"),
        # the headline source build
        dict(name="aknn_million", kind="aknn", n=1_000_000, d=128, data="mixture", metric="l2"),
        # the graph build of a mid-sized index
        dict(name="graph", kind="graph", n=200_000, d=128, data="mixture", metric="l2"),
        # thresholds and ground truth for an evaluation, long rows
        dict(name="truth", kind="truth", n=100_000, d=300, data="unit", metric="l2", nq=2_000),
        # the verifier of a mid-sized index
        dict(name="verifier", kind="verifier", n=250_000),
        # a training step on the sampled rows
        dict(name="objective", kind="objective", n=120_000, nk=100, m=8, cs=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "aknn", "aknn", "graph", "truth", "verifier", "objective"])
    data = rng.choice(["mixture", "unit"])
    metric = "ip" if data == "unit" and rng.random() < 0.4 else "l2"
    if kind == "verifier":
        return dict(kind=kind, n=_log(rng, 3_000, 400_000))
    if kind == "objective":
        return dict(kind=kind, n=_log(rng, 1_000, 120_000), nk=rng.randint(16, 128), m=rng.randint(2, 16),
                    cs=rng.randint(16, 256))
    d = rng.choice([8, 32, 96, 100, 128, 128, _log(rng, 8, 400)])
    if kind == "query":
        if rng.random() < 0.1:
            d = 960
        return dict(kind=kind, n=min(_log(rng, 2_000, 200_000), 24_000_000 // d), d=d, data=data, metric=metric,
                    nq=_log(rng, 1, 10_000), k=rng.choice([0, *KS]), L=rng.choice([0, 128, _log(rng, 20, 600)]),
                    call=rng.choice(["host", "graph"]), pinned=rng.random() < 0.5)
    if kind == "aknn":
        return dict(kind=kind, n=min(_log(rng, 1_500, 250_000), 16_000_000 // d), d=d, data=data, metric=metric)
    if kind == "graph":
        return dict(kind=kind, n=min(_log(rng, 2_000, 200_000), 16_000_000 // d), d=min(d, 254), data=data,
                    metric="l2")
    return dict(kind="truth", n=min(_log(rng, 2_000, 100_000), 16_000_000 // d), d=d, data=data, metric=metric,
                nq=_log(rng, 50, 2_000))


# ------------------------------------------------------------------ inputs


def _rows(case, seed, extra):
    """Base rows and `extra` query rows (host arrays) of one distribution."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 1)
    n, d = case["n"] + extra, case["d"]
    if case["data"] == "unit":
        x = torch.randn((n, d), generator=g, device="cuda")
        x /= x.norm(dim=1, keepdim=True)
    else:
        centers = torch.rand((1000, d), generator=g, device="cuda") * 128.0
        x = torch.randn((n, d), generator=g, device="cuda")
        x.mul_(20.0).add_(centers[torch.randint(1000, (n,), generator=g, device="cuda")])
        x.clamp_(0.0, 255.0).round_()
    return x[:case["n"]].cpu().numpy(), x[case["n"]:].cpu().numpy()


def _cutoffs(n, nk, seed):
    """Ascending squared cutoffs of n rows: r^2 (i / nk)^(2 / dim) with the row's
    radius and local dimension, plus spacing noise, as AKNN lists have them."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 3)
    dim = 8.0 + 24.0 * torch.rand((n, 1), generator=g, device="cuda", dtype=torch.float64)
    rad = 60_000.0 * torch.exp(0.15 * torch.randn((n, 1), generator=g, device="cuda", dtype=torch.float64))
    gap = torch.empty((n, nk), device="cuda", dtype=torch.float64).exponential_(generator=g)
    pos = torch.cumsum(gap, dim=1) / nk
    return (rad * pos.pow(2.0 / dim)).round().float()


def _index(ctx, case, base):
    """Builds the whole index over `base` and makes it resident."""
    from anqi import lrq_fit, pipeline
    metric = case["metric"]
    ids, keys, _ = pipeline.aknn_build(ctx, base, metric=metric)
    mu, basis, cb = (np.asarray(a, np.float32) for a in lrq_fit.train_gpu(keys, len(keys), log=lambda s: None))
    coeff, codes = ctx.lrq_encode(keys, mu, basis, cb)
    lifted, m2, sc = ctx.lift(base, keys[:, -1], metric=metric)
    deg, links, tree, _ = pipeline.graph_build(ctx, lifted, ids)
    ctx.index_load(base, lifted, deg, links, tree, sc, m2, metric=metric)
    ctx.verifier_load_bits(coeff, codes.reshape(-1), None, codes.shape[1], mu, basis, cb, 8,
                           signed_keys=metric == "ip")
    for k in KS:
        ctx.verifier_materialize(k)


def _csr_rows(case, k):
    """Room for a ground-truth CSR: k results a query on average."""
    return 1024 + 2 * k * case["nq"]


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed):
    from anqi import pipeline
    from anqi._lib import Context
    kind = case["kind"]
    s = dict(case)
    if kind == "objective":
        n, nk, m, cs = (case[x] for x in ("n", "nk", "m", "cs"))
        T = _cutoffs(n, nk, seed).double()
        mu = T.mean(dim=0)
        G = torch.linalg.eigh((T - mu).T @ (T - mu))[1][:, -min(m, nk):].T.contiguous()
        res = T - (mu + ((T - mu) @ G.T) @ G)
        q = torch.linspace(0.0, 1.0, cs, dtype=torch.float64, device="cuda")
        B = torch.quantile(res[:: max(1, n // 4000)], q, dim=0).T.contiguous()
        s.update(T=T, mu=mu.requires_grad_(), G=G.requires_grad_(), B=B.requires_grad_())
        return s
    ctx = s["ctx"] = Context(0)
    if kind == "verifier":
        s["keys"] = _cutoffs(case["n"], 100, seed).cpu().numpy()
        return s
    nq = case.get("nq", 0)
    base, query = _rows(case, seed, nq)
    if kind == "aknn":
        s["base"] = base
    elif kind == "graph":
        s["warm"], keys, _ = pipeline.aknn_build(ctx, base)
        s["lifted"] = ctx.lift(base, keys[:, -1])[0]
    elif kind == "truth":
        s["hints"] = pipeline.aknn_build(ctx, base, metric=case["metric"])[0]
        s.update(base=base, query=query)
    else:
        rng = np.random.default_rng(int(seed))
        k, L = case["k"], case["L"]
        if not k:
            k = rng.choice(np.array(KS, np.uint32), size=nq)
        if not L:
            L = rng.integers(64, 601, size=nq).astype(np.uint32)
        _index(ctx, case, base)
        # the buffers a serving loop receives its results in, pinned or plain
        sizes = (nq + 1, 1024 + 128 * nq, nq)
        if case["pinned"]:
            pq = _pinned(query.shape, torch.float32)
            pq[:] = query
            query = pq
            out = tuple(_pinned(c, torch.int32).view(np.uint32) for c in sizes)
        else:
            out = tuple(np.empty(c, np.uint32) for c in sizes)
        out[1][:] = 0
        s.update(query=query, ks=k, Ls=L, out=out)
    return s


# --------------------------------------------------------------- one pass


def _kept(state, name, a, rows):
    """`a` in a buffer of `rows` rows that the program keeps (zeros past its end),
    so that results of any length have one shape."""
    buf = state.get("kept " + name)
    if buf is None:
        buf = state["kept " + name] = np.zeros((rows, *a.shape[1:]), a.dtype)
    m = min(rows, len(a))
    buf[:m] = a[:m]
    return buf


def run(state):
    from anqi import lrq_fit, lrq_torch, pipeline
    kind = state["kind"]
    if kind == "objective":
        mu, G, B = state["mu"], state["G"], state["B"]
        mu.grad = G.grad = B.grad = None
        loss, codes = lrq_torch.lrq_loss(state["T"], mu, G, B)
        loss.backward()
        return dict(loss=loss.detach(), codes=codes, g_mu=mu.grad, g_G=G.grad, g_B=B.grad)
    ctx = state["ctx"]
    if kind == "query":
        if state["call"] == "graph":
            ctx.query_upload(state["query"], state["ks"], state["Ls"])
            ctx.query_run_graph()
            r = ctx.query_download()
        else:
            r = ctx.rknn_query(state["query"], state["ks"], state["Ls"], keep_candidates=state["metric"] == "ip",
                               out=state["out"])
        ids = state["out"][1]
        if len(r.pred_ids) and not np.may_share_memory(r.pred_ids, ids):
            m = min(len(ids), len(r.pred_ids))
            ids[:m] = r.pred_ids[:m]
        found = dict(off=r.pred_off, ids=ids, n_dist=r.n_dist)
        if r.cand_off is not None:
            found.update(cand_off=r.cand_off, cand_ids=_kept(state, "cand", r.cand_ids, 4 * len(ids)))
        return found
    if kind == "aknn":
        ids, keys, _ = pipeline.aknn_build(ctx, state["base"], metric=state["metric"])
        return dict(ids=ids, keys=keys)
    if kind == "graph":
        deg, links, tree, _ = pipeline.graph_build(ctx, state["lifted"], state["warm"])
        rows = state["n"] // 10 + 64
        return dict(deg=deg, links=links, indices=_kept(state, "indices", tree.indices, state["n"]),
                    left=_kept(state, "left", tree.left, rows), right=_kept(state, "right", tree.right, rows),
                    hyperplane=_kept(state, "hyperplane", tree.hyperplane, rows))
    if kind == "truth":
        base, query, metric = state["base"], state["query"], state["metric"]
        ids, keys = pipeline.exact_thresholds(ctx, base, 100, method="tc", hints=state["hints"], metric=metric)
        csr = []
        for k in KS:
            off, found, key = pipeline.rknn_ground_truth(ctx, base, query, keys[:, k - 1], method="tc", metric=metric)
            rows = _csr_rows(state, k)
            csr.append([off, _kept(state, f"ids{k}", found, rows), _kept(state, f"keys{k}", key, rows)])
        return dict(ids=ids, keys=keys, csr=csr)
    keys = state["keys"]
    mu, basis, cb = lrq_fit.train_gpu(keys, len(keys), log=lambda s: None)
    f = [np.asarray(a, np.float32) for a in (mu, basis, cb)]
    coeff, codes = ctx.lrq_encode(keys, *f)
    thr = [ctx.lrq_materialize(coeff, codes, *f, k) for k in KS]
    return dict(mu=mu, basis=basis, codebook=cb, coeff=coeff, codes=codes, thr=thr)


# ------------------------------------------------------------------- work


def work(case):
    """Inputs read once, outputs written once.  A query evaluates about eight
    lifted rows per beam entry; a batch reads each index row at most once.  The
    exact stages cannot do without a product per pair; the approximate source
    build without the pairs of one leaf (500 rows) per row."""
    kind = case["kind"]
    if kind == "objective":
        n, nk, m, cs = (case[x] for x in ("n", "nk", "m", "cs"))
        return dict(bytes=8.0 * n * nk + n * nk + 16.0 * (nk + m * nk + nk * cs), flops=8.0 * n * nk * m + 10.0 * n * nk)
    n = case["n"]
    if kind == "verifier":
        return dict(bytes=n * (400.0 + 32 + 100 + 12), flops=8.0 * 12 * min(n, 120_000) * 100 * 100)
    d = case["d"]
    if kind == "query":
        L = case["L"] or 332
        rows = 8.0 * L * case["nq"]
        per_row = 4.0 * (d + 2)
        return dict(bytes=min(rows * per_row, n * (per_row + 4.0 * 48)) + case["nq"] * 4.0 * d, flops=rows * 3.0 * (d + 2))
    if kind == "aknn":
        return dict(bytes=4.0 * n * d + 800.0 * n, flops=2.0 * n * min(n, 500) * d)
    if kind == "graph":
        return dict(bytes=4.0 * n * (d + 2) + 400.0 * n + 196.0 * n, flops=3.0 * n * 100 * (d + 2))
    return dict(bytes=4.0 * (n + case["nq"]) * d + 800.0 * n, flops=2.0 * n * (n + 3.0 * case["nq"]) * d)


# ------------------------------------------------------------------ exact


def exact(case, seed):
    """64-bit values of the computed outputs; lists found by an approximate
    build and results that are ids have none."""
    kind = case["kind"]
    if kind == "objective":
        s = prepare(case, seed)
        T, mu, G, B = s["T"], s["mu"], s["G"], s["B"]
        c = (T - mu) @ G.T
        res = (T - (mu + c @ G)).detach()
        codes = torch.empty(res.shape, dtype=torch.int64, device="cuda")
        edges = (B[:, 1:] + B[:, :-1]).detach() * 0.5
        for j in range(T.shape[1]):
            codes[:, j] = torch.searchsorted(edges[j].contiguous(), res[:, j].contiguous())
        r = mu + c @ G + torch.gather(B, 1, codes.T).T - T
        loss = r.square().mean()
        loss.backward()
        return dict(loss=loss.detach(), codes=None, g_mu=mu.grad, g_G=G.grad, g_B=B.grad)
    if kind != "truth":
        return None
    base, query = (torch.from_numpy(a).cuda().double() for a in _rows(case, seed, case["nq"]))
    n, ip = len(base), case["metric"] == "ip"
    norm = base.square().sum(dim=1)

    def keys_of(x):
        dot = x @ base.T
        return -dot if ip else x.square().sum(dim=1, keepdim=True) + norm - 2.0 * dot

    keys = torch.empty((n, 100), dtype=torch.float64, device="cuda")
    for at in range(0, n, 4096):
        part = keys_of(base[at:at + 4096])
        rows = torch.arange(len(part), device="cuda")
        part[rows, at + rows] = math.inf
        keys[at:at + 4096] = torch.topk(part, 100, dim=1, largest=False, sorted=True)[0]
    csr = []
    for k in KS:
        found = []
        for at in range(0, len(query), 1024):
            for row in keys_of(query[at:at + 1024]):
                found.append(torch.sort(row[row <= keys[:, k - 1]])[0])
        room = torch.zeros(_csr_rows(case, k), dtype=torch.float64, device="cuda")
        found = torch.cat(found)[:len(room)]
        room[:len(found)] = found
        csr.append([None, None, room])
    return dict(ids=None, keys=keys, csr=csr)
