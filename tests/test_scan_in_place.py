"""The scan with its output in its input, as the grid build calls it."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 4095, 4097, 40 * 4096 + 3, 3_000_001])
@pytest.mark.parametrize("inclusive", [0, 1])
def test_scan_in_place(n, inclusive):
    import torch
    import photonmap
    a = np.random.default_rng(n).integers(0, 200, n).astype(np.int32)
    want = np.cumsum(a, dtype=np.int64) - (0 if inclusive else a)
    ctx = photonmap.Context(0)
    x = torch.from_numpy(a).cuda()
    torch.cuda.synchronize()
    ctx._check(ctx.L.pm_scan_u32(ctx.h, x.data_ptr(), x.data_ptr(), n, inclusive), "pm_scan_u32")
    assert np.array_equal(x.cpu().numpy(), want)
    assert ctx.status() == 0
    ctx.close()
