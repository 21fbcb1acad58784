"""The LRQ objective's gradients with an infinite residual: infinite where the
formula is, not a number only where it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nk", [(1, 20), (1, 128), (12, 40)])
def test_infinite_residual(m, nk):
    import torch

    from anqi._lib import load_library

    rng = np.random.default_rng(m + nk)
    n, cs, scale = 300, 16, 0.5
    T, r, c = rng.standard_normal((n, nk)), rng.standard_normal((n, nk)), rng.standard_normal((n, m))
    mu, a = rng.standard_normal(nk), rng.integers(0, cs, (n, nk)).astype(np.uint8)
    G = np.abs(rng.standard_normal((m, nk)))  # one sign: infinities of one sign in every sum but the row's own column
    T = np.abs(T) + 5
    r[137, 3] = np.inf
    with np.errstate(invalid="ignore"):
        s = r @ G.T
        g_mu = scale * (r.sum(0) - s.sum(0) @ G)
        g_G = scale * (c.T @ r + s.T @ (T - mu))
        g_B = np.zeros((nk, cs))
        for k in range(nk):
            np.add.at(g_B[k], a[:, k], scale * r[:, k])
    dev = [torch.from_numpy(v).cuda() for v in (T, mu, G, r, c, a)]
    out = [torch.empty(v.shape, dtype=torch.float64, device="cuda") for v in (g_mu, g_G, g_B)]
    p = [v.data_ptr() for v in dev + out]
    assert load_library().anqi_lrq_objective_backward(p[0], n, nk, m, p[1], p[2], p[3], p[4], p[5], cs, scale, p[6],
                                                      p[7], p[8], torch.cuda.current_stream().cuda_stream) == 0
    for got, want in zip(out, (g_mu, g_G, g_B)):
        got = got.cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.allclose(got, want, rtol=1e-11, atol=1e-11, equal_nan=True)
    assert np.isinf(g_mu).sum() == nk - 1
