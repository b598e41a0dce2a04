"""Attention with one key head, whose (token, head) pairs are the rows of the key-loop form: suffix batches around the
size where it takes over from the cluster form, ragged row counts, masked keys, and single suffixes of the cluster form, against
a plain fp32 reference."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,l,keys,h,d", [(3, 50, 594, 8, 256), (4, 50, 594, 8, 256), (9, 50, 641, 8, 256), (32, 50, 994, 8, 256),
                                          (40, 1, 130, 3, 256), (17, 128, 257, 5, 256), (2, 129, 129, 7, 256), (2, 33, 200, 8, 128),
                                          # output columns split over two clusters per head, or not: around the clusters that fit
                                          (1, 50, 896, 8, 256), (1, 50, 1018, 8, 256), (1, 56, 1018, 7, 256), (1, 7, 1024, 8, 256)])
def test_one_key_head_matches_fp32(b, l, keys, h, d):
    from tybok_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(b + l)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)  # noqa: E731
    q, k, v = rnd(b * l, h * d), rnd(b, 1, keys + 5, d), rnd(b, 1, keys + 5, d)
    valid = torch.ones(b, keys, dtype=torch.uint8, device="cuda")
    valid[:, keys // 3 : keys // 2] = 0
    y, yp = ops.attention(q, k, v, valid, tokens=l, keys=keys, scale=d**-0.5, out_planes=True, out_shift=6)
    ops.check_status()
    s = torch.einsum("blhd,bkd->blhk", q.view(b, l, h, d).float(), k[:, 0, :keys].float()) * d**-0.5
    p = s.masked_fill(valid[:, None, None, :] == 0, float("-inf")).softmax(-1)
    ref = torch.einsum("blhk,bkd->blhd", p, v[:, 0, :keys].float()).reshape(b * l, h * d)
    assert float((y.float() - ref).norm() / ref.norm()) <= 6e-3
    planes = yp.view(torch.float8_e5m2).float().sum(0)
    assert float((planes - y.float() * 64).abs().max()) <= 2.0**-16
