"""RMS / AdaRMS rows with two vectors per thread: widths that leave the last threads one vector or none, single rows, and row
counts on both sides of a group of modulation rows, every output form against fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,w", [(1, 264), (3, 520), (50, 1024), (51, 1160), (128, 2048), (300, 4088), (7, 4096)])
@pytest.mark.parametrize("ada", [False, True])
def test_rows(m, w, ada):
    from tybok_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(m + w)
    x = torch.empty(m, w, device="cuda").normal_(0, 2, generator=g).bfloat16()
    groups = (m + 49) // 50
    a = torch.empty(groups, 2 * w, device="cuda").normal_(0, 1, generator=g) if ada else torch.empty(w, device="cuda").normal_(0, 1, generator=g)
    x32 = x.float()
    n = x32 * torch.rsqrt(x32.pow(2).mean(-1, keepdim=True) + 1e-6)
    if ada:
        row = a.repeat_interleave(50, 0)[:m]
        ref = n * (1 + row[:, :w]) + row[:, w:]
    else:
        ref = n * (1 + a)
    lib, s = _lib.load(), torch.cuda.current_stream().cuda_stream
    wt, mod = (None, a.data_ptr()) if ada else (a.data_ptr(), None)
    y, pl = torch.empty_like(x), torch.empty(3, m, w, dtype=torch.uint8, device="cuda")
    assert lib.tybok_rmsnorm(x.data_ptr(), w, wt, mod, 2 * w, 50, m, w, 1e-6, y.data_ptr(), w, pl.data_ptr(), 4, s) == 0
    p2, rs = torch.empty(2, m, w, dtype=torch.uint8, device="cuda"), torch.empty(m, device="cuda")
    assert lib.tybok_norm_planes2(x.data_ptr(), w, 1 if ada else 0, a.data_ptr(), None, 2 * w, 50, m, w, 1e-6, p2.data_ptr(), rs.data_ptr(), s) == 0
    ops.check_status()
    assert float((y.float() - ref).norm() / ref.norm()) <= 4e-3
    assert float((pl.view(torch.float8_e5m2).float().sum(0) / 16 - y.float()).abs().max()) <= 2.0**-20
    two = p2.view(torch.float8_e4m3fn).float().sum(0) * rs[:, None]
    assert float((two - y.float()).abs().max()) <= 1e-5 * float(y.float().abs().max())
