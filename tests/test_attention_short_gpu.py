"""head_dim 128 with up to 64 query rows (every row twice in the Q tile, P half through shared memory): row counts around
a quadrant and the limit, key counts around a block, masked keys, and scores that grow from block to block so that rows are
rescaled, against a plain fp32 reference."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("b,l,keys,h,g", [(1, 1, 1, 2, 2), (2, 32, 64, 3, 3), (1, 33, 65, 4, 2), (3, 50, 129, 2, 2), (1, 64, 640, 24, 24),
                                          (1, 50, 4146, 24, 24), (2, 65, 129, 2, 2), (5, 16, 300, 4, 1)])
def test_matches_fp32(b, l, keys, h, g, grow):
    from tybok_b200 import ops

    d = 128
    gen = torch.Generator(device="cuda").manual_seed(l + keys)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=gen)  # noqa: E731
    q, k, v = rnd(b * l, h * d).bfloat16(), rnd(b, g, keys + 3, d), rnd(b, g, keys + 3, d).bfloat16()
    if grow:
        k *= torch.linspace(0.1, 6.0, keys + 3, device="cuda")[:, None]
    k = k.bfloat16()
    valid = torch.ones(b, keys, dtype=torch.uint8, device="cuda")
    valid[:, keys // 3 : keys // 2] = 0
    y, yp = ops.attention(q, k, v, valid, tokens=l, keys=keys, scale=d**-0.5, out_planes=True, out_shift=6)
    ops.check_status()
    kk, vv = (t[:, :, :keys].float().repeat_interleave(h // g, 1) for t in (k, v))
    s = torch.einsum("blhd,bhkd->bhlk", q.view(b, l, h, d).float(), kk) * d**-0.5
    p = s.masked_fill(valid[:, None, None, :] == 0, float("-inf")).softmax(-1)
    ref = torch.einsum("bhlk,bhkd->blhd", p, vv).reshape(b * l, h * d)
    assert float((y.float() - ref).norm() / ref.norm()) <= 6e-3
    planes = yp.view(torch.float8_e5m2).float().sum(0)
    assert float((planes - y.float() * 64).abs().max()) <= 2.0**-16
