"""Calls of different sizes on several threads at once: the shared memory one of
them asks for is no limit to another's launch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_objective_on_two_threads():
    import torch

    from anqi._lib import load_library

    lib = load_library()
    failed, start = [], threading.Barrier(2)

    def work(nk, cs, n=64, m=4, calls=3000):
        g = torch.Generator(device="cuda").manual_seed(cs)
        f = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        T, mu, G, B = f(n, nk), f(nk), f(m, nk), f(nk, cs).sort(dim=1).values.contiguous()
        r, c, a, loss = f(n, nk), f(n, m), torch.zeros((n, nk), dtype=torch.uint8, device="cuda"), f(1)
        g_mu, g_G, g_B = f(nk), f(m, nk), f(nk, cs)
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        start.wait()
        for _ in range(calls):
            rc = lib.anqi_lrq_objective_forward(T.data_ptr(), n, nk, m, mu.data_ptr(), G.data_ptr(), B.data_ptr(), cs,
                                                None, r.data_ptr(), c.data_ptr(), a.data_ptr(), loss.data_ptr(),
                                                s.cuda_stream)
            rc |= lib.anqi_lrq_objective_backward(T.data_ptr(), n, nk, m, mu.data_ptr(), G.data_ptr(), r.data_ptr(),
                                                  c.data_ptr(), a.data_ptr(), cs, 2.0, g_mu.data_ptr(), g_G.data_ptr(),
                                                  g_B.data_ptr(), s.cuda_stream)
            if rc:
                failed.append((nk, cs, rc))
                break
        s.synchronize()

    threads = [threading.Thread(target=work, args=a) for a in ((100, 256), (8, 16))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_builds_on_two_contexts():
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(9)
    cases = [(rng.standard_normal((2500, 24)).astype(np.float32), dict(k=20, ef=600, trees=4, leaf=60)),
             (rng.standard_normal((2500, 200)).astype(np.float32), dict(k=100, ef=200, trees=4, leaf=400))]
    want, got = [], [[], []]
    for x, opts in cases:
        with Context(0) as ctx:
            want.append(pipeline.aknn_build(ctx, x, **opts))

    def work(i):
        with Context(0) as ctx:
            for _ in range(15):
                got[i].append(pipeline.aknn_build(ctx, cases[i][0], **cases[i][1]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert len(got[i]) == 15
        for g in got[i]:
            assert np.array_equal(g[0], want[i][0])
            assert np.array_equal(g[1].view(np.uint32), want[i][1].view(np.uint32))
