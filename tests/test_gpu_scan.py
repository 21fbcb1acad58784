"""The whole-matrix scan (csrc/tc.cu tc_scan_kernel) at its tile edges, against
the FP32 CUDA-core ground truth: same ids, same key bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# base tiles of 256 rows and query tiles of 128 with one row over and under,
# one K chunk to sixteen, the last chunk partial (d = 20, 72), the query tile
# resident (up to 512 padded) and streamed, exact-integer rows, thresholds that
# keep every pair, none and some
@pytest.mark.parametrize("n,nq,d,kind,metric", [
    (255, 1, 20, "float", "l2"),
    (256, 128, 64, "int", "l2"),
    (257, 129, 72, "float", "ip"),
    (1025, 127, 128, "int", "l2"),
    (700, 33, 512, "float", "l2"),
    (513, 130, 520, "float", "ip"),
    (400, 40, 1024, "float", "l2"),
])
def test_scan_equals_fp32(n, nq, d, kind, metric):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n + nq, d))
    x = (np.rint(20 * x) if kind == "int" else x).astype(np.float32)
    x[7] = x[3]
    base, query = np.ascontiguousarray(x[:n]), np.ascontiguousarray(x[n:])
    bits = lambda a: a.view(np.uint32)  # noqa: E731
    with Context(0) as ctx:
        want = pipeline.exact_thresholds(ctx, base, 100, metric=metric)
        got = pipeline.exact_thresholds(ctx, base, 100, method="tc", metric=metric)
        assert np.array_equal(got[0], want[0]) and np.array_equal(bits(got[1]), bits(want[1]))
        inf = np.float32(np.inf)
        mixed = want[1][:, 49].copy()
        mixed[::3], mixed[1::7] = inf, -inf
        for rk2 in (want[1][:, 99], mixed, np.full(n, -inf, np.float32)):
            w = pipeline.rknn_ground_truth(ctx, base, query, rk2, metric=metric)
            g = pipeline.rknn_ground_truth(ctx, base, query, rk2, method="tc", metric=metric)
            assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])
            assert np.array_equal(bits(g[2]), bits(w[2]))
