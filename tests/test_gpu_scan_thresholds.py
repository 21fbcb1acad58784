"""The whole-matrix scan with thresholds of any finite size: same result as the FP32
form, and a few huge ones do not make it test every pair one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return a.view(np.uint32)


@pytest.mark.parametrize("n,nq,d,kind,metric", [
    (700, 130, 72, "float", "l2"), (1025, 127, 128, "int", "l2"), (600, 90, 100, "float", "ip"),
])
def test_scan_thresholds_equal_fp32(n, nq, d, kind, metric):
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n + nq, d))
    x = (np.rint(20 * x) if kind == "int" else x).astype(np.float32)
    base, query = np.ascontiguousarray(x[:n]), np.ascontiguousarray(x[n:])
    top = np.finfo(np.float32).max
    with Context(0) as ctx:
        exact = pipeline.exact_thresholds(ctx, base, 100, metric=metric)[1]
        for values in ([top], [-top], [top, -top, 1e30, -1e30, 1e10, 0.0, np.inf]):
            rk2 = exact[:, 49].copy()
            for t, v in enumerate(values):
                rk2[5 + t :: 40] = v
            w = pipeline.rknn_ground_truth(ctx, base, query, rk2, metric=metric)
            g = pipeline.rknn_ground_truth(ctx, base, query, rk2, method="tc", metric=metric)
            assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])
            assert np.array_equal(bits(g[2]), bits(w[2]))


def scan_us(run):
    from torch.profiler import ProfilerActivity, profile

    run()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
    return sum(e.device_time_total for e in p.key_averages() if "tc_scan_kernel" in e.key)


def test_one_huge_threshold_costs_one_column():
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(3)
    n, nq, d = 40_000, 1000, 64
    base = rng.standard_normal((n, d)).astype(np.float32)
    query = rng.standard_normal((nq, d)).astype(np.float32)
    with Context(0) as ctx:
        rk2 = pipeline.exact_thresholds(ctx, base, 10, method="tc")[1][:, 9].copy()
        huge = rk2.copy()
        huge[n // 2] = np.finfo(np.float32).max
        plain_us = scan_us(lambda: pipeline.rknn_ground_truth(ctx, base, query, rk2, method="tc"))
        huge_us = scan_us(lambda: pipeline.rknn_ground_truth(ctx, base, query, huge, method="tc"))
    assert 0 < plain_us and huge_us < 2 * plain_us
