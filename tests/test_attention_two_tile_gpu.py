"""Self- and cross-attention at head_dim 128 around the size where a CTA takes two query tiles: last pairs with one tile or
a few rows, ragged and fully masked key blocks, several batch elements, growing row maxima; against a plain fp32 reference."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,l,keys,h,g", [(1, 768, 768, 24, 24), (1, 769, 1, 24, 24), (1, 897, 127, 24, 24), (1, 1030, 385, 24, 24),
                                          (2, 400, 513, 24, 24), (3, 1281, 300, 6, 2), (1, 4146, 129, 24, 24)])
def test_two_tile_form_matches_fp32(b, l, keys, h, g):
    from tybok_b200 import ops

    d = 128
    gen = torch.Generator(device="cuda").manual_seed(l + keys)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=gen).to(torch.bfloat16)  # noqa: E731
    q, k, v = rnd(b * l, h * d), rnd(b, g, keys + 3, d), rnd(b, g, keys + 3, d)
    k *= torch.linspace(0.2, 6.0, keys + 3, device="cuda").to(torch.bfloat16)[None, None, :, None]  # maxima that keep growing
    valid = torch.ones(b, keys, dtype=torch.uint8, device="cuda")
    if keys > 300:
        valid[:, :128] = 0  # a whole block
        valid[0, 200:290] = 0
    elif keys > 1:
        valid[:, keys // 2 : keys // 2 + 9] = 0
    y, yp = ops.attention(q, k, v, valid, tokens=l, keys=keys, scale=d**-0.5, out_planes=True, out_shift=6)
    ops.check_status()
    kk, vv = (t[:, :, :keys].float().repeat_interleave(h // g, dim=1) for t in (k, v))
    s = (q.view(b, l, h, d).transpose(1, 2).float() @ kk.transpose(-1, -2)) * d**-0.5
    p = s.masked_fill(valid[:, None, None, :] == 0, float("-inf")).softmax(-1)
    ref = (p @ vv).transpose(1, 2).reshape(b * l, h * d)
    assert float((y.float() - ref).norm() / ref.norm()) <= 6e-3
    assert float((yp.view(torch.float8_e5m2).float().sum(0) - y.float() * 64).abs().max()) <= 2.0**-16
