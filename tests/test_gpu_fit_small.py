"""The fit's column sort around one tile (4,096 values): a column that fits is sorted
in one launch, and both forms put NaN last, as NumPy does."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nk", [(2, 3), (33, 128), (1025, 4), (4096, 5), (4097, 5)])
def test_sort_form_and_order(m, nk):
    import torch
    from torch.profiler import ProfilerActivity, profile

    from anqi._lib import load_library

    lib = load_library()
    x = np.random.default_rng(m).standard_normal((nk, m))
    x[:, :: max(2, m // 7)] = np.nan
    x[-1, 1:] = np.inf
    res = torch.from_numpy(x.reshape(-1).copy()).cuda()
    scr = torch.empty(int(lib.anqi_lrq_fit_codebooks_scratch(m, nk)), dtype=torch.float64, device="cuda")
    cb = torch.empty(nk * 2, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        assert lib.anqi_lrq_fit_codebooks(res.data_ptr(), m, nk, 2, 1, scr.data_ptr(), scr.numel(), cb.data_ptr(),
                                          stream) == 0
        torch.cuda.synchronize()
    ran = {e.key: e.count for e in p.key_averages()}
    count = lambda name: sum(c for k, c in ran.items() if re.search(name, k))  # noqa: E731
    assert count("fit_sort_small_kernel") == (m <= 4096) and count("fit_sort_move_kernel") == 8 * (m > 4096)
    assert np.array_equal(scr[: nk * m].cpu().numpy().reshape(nk, m), np.sort(x, axis=1), equal_nan=True)
