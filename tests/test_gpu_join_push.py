"""LocalJoin's pushes, 32 candidates at a time, against the oracle's one by one:
same heaps, same value bits, same update counts."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


# heaps below, at and past a warp's width; samples past 32 (lists without masks);
# integer rows (ties at the heap's top); heaps whose stored values are not the
# distances, so that an entry thrown out comes back with another value
@pytest.mark.parametrize("n,d,K,sample,kind", [
    (1500, 12, 50, 20, "plain"),
    (1200, 5, 31, 32, "int"),
    (900, 33, 32, 20, "loose"),
    (1200, 16, 65, 48, "loose"),
    (700, 8, 7, 7, "int"),
])
def test_join_equals_oracle(n, d, K, sample, kind):
    from anqi._lib import Context

    rng = np.random.default_rng(n + K)
    x = rng.standard_normal((n, d))
    if kind == "int":
        x = np.rint(2 * x)
    x = np.ascontiguousarray(x, np.float32)
    nrm = ol.norms(x)
    cand = rng.integers(0, n, size=(n, 2 * K)).astype(np.uint32)
    ids, vals = ol.warm_start(x, nrm, cand, 2 * K, K)
    if kind == "loose":
        order = np.argsort(-vals, axis=1, kind="stable")
        ids = np.ascontiguousarray(np.take_along_axis(ids, order, 1))
        vals = np.take_along_axis(vals, order, 1) * rng.choice([1.0, 1.5], size=(n, K))
        vals = np.ascontiguousarray(-np.sort(-vals, axis=1), np.float32)
    want = ol.localjoin(x, nrm, ids, vals, sample=sample)
    with Context(0) as ctx:
        for precision in (0, 1) if sample <= 32 else (0,):
            gi, gv = ids.copy(), vals.copy()
            up = np.zeros(6, np.uint64)
            done, ms = C.c_uint32(), C.c_float()
            ctx._check(ctx.lib.anqi_graph_localjoin_precision(ctx.h, x, n, d, K, sample, 6, precision, gi, gv, up,
                                                              C.byref(done), C.byref(ms)), "localjoin")
            assert [int(u) for u in up[:done.value]] == want[2]
            assert np.array_equal(gi, want[0])
            assert np.array_equal(gv.view(np.uint32), want[1].view(np.uint32))
