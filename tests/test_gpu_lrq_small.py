"""The LRQ objective's backward where a warp has one row or none and a block all rows
of a column: gradients against the formula, overwriting what was there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one row, a block's warps (12, or 8 past rank 8) and one over, the codebook
# gradient's 64 rows a block and one over; column groups with and without a tail
@pytest.mark.parametrize("n,nk,m,cs", [
    (1, 1, 1, 1), (8, 33, 9, 7), (9, 40, 16, 256), (12, 128, 8, 256), (13, 100, 8, 16), (64, 31, 3, 64), (65, 97, 8, 256),
])
def test_backward_of_few_rows(n, nk, m, cs):
    import torch

    from anqi._lib import load_library

    rng = np.random.default_rng(n + nk)
    T, r, c = rng.standard_normal((n, nk)), rng.standard_normal((n, nk)), rng.standard_normal((n, m))
    mu, G, a = rng.standard_normal(nk), rng.standard_normal((m, nk)), rng.integers(0, cs, (n, nk)).astype(np.uint8)
    s = r @ G.T
    want = [2 * (r.sum(0) - s.sum(0) @ G), 2 * (c.T @ r + s.T @ (T - mu)), np.zeros((nk, cs))]
    for k in range(nk):
        np.add.at(want[2][k], a[:, k], 2 * r[:, k])
    dev = [torch.from_numpy(v).cuda() for v in (T, mu, G, r, c, a)]
    out = [torch.full(v.shape, np.nan, dtype=torch.float64, device="cuda") for v in want]
    p = [v.data_ptr() for v in dev + out]
    assert load_library().anqi_lrq_objective_backward(p[0], n, nk, m, p[1], p[2], p[3], p[4], p[5], cs, 2.0, p[6], p[7],
                                                      p[8], torch.cuda.current_stream().cuda_stream) == 0
    # sums of at most n nk products of size 1 to 10: a few hundred roundings of 1e-16
    for got, w in zip(out, want):
        assert np.allclose(got.cpu().numpy(), w, rtol=1e-11, atol=1e-10)
