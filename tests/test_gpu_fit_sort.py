"""The fit's column sort: the sorted columns it leaves at the front of its scratch
against NumPy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# around a warp's 32 and 512 keys and a tile's 4,096; one column and the most;
# ties, both zeros, subnormals, infinities, every exponent and one
@pytest.mark.parametrize("m,nk,kind", [
    (2, 1, "normal"), (31, 3, "wide"), (511, 2, "ties"), (513, 128, "normal"), (4095, 1, "wide"), (4096, 3, "ties"),
    (4097, 2, "normal"), (20_001, 5, "wide"), (12_289, 100, "narrow"),
])
def test_columns_sorted(m, nk, kind):
    import torch

    from anqi._lib import load_library

    rng = np.random.default_rng(m + nk)
    x = rng.standard_normal((nk, m))
    if kind == "ties":
        x = np.rint(2 * x) * 0.5
        x[:, ::7] = -0.0
    elif kind == "wide":
        x *= 10.0 ** rng.uniform(-320, 300, (nk, m))
        x[0, : m // 4] = np.inf
        x[0, m // 4 : m // 3] = -np.inf
    elif kind == "narrow":
        x = 1.5 + 1e-12 * x
    lib = load_library()
    res = torch.from_numpy(x.reshape(-1).copy()).cuda()
    scr = torch.empty(int(lib.anqi_lrq_fit_codebooks_scratch(m, nk)), dtype=torch.float64, device="cuda")
    cb = torch.empty(nk * 2, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.anqi_lrq_fit_codebooks(res.data_ptr(), m, nk, 2, 1, scr.data_ptr(), scr.numel(), cb.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert np.array_equal(scr[: nk * m].cpu().numpy().reshape(nk, m), np.sort(x, axis=1))
    assert np.array_equal(res.cpu().numpy(), x.reshape(-1))
