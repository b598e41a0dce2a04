"""Masked keys in every attention form: rows that meet masked keys only, for a block or for all of them, at every scale that the entry
takes; the images with the tuning aids against those without, the same bits; and blocks of small weight in the merge."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# suffix over key blocks (rows pushed, and staged in L2), one block, the key loop at both head sizes, up to 64 rows, two tiles
FORMS = [(1, 50, 594, 8, 1, 256), (2, 50, 594, 8, 2, 256), (1, 50, 100, 8, 1, 256), (1, 300, 300, 8, 1, 256), (1, 106, 400, 3, 3, 128),
         (1, 50, 700, 24, 24, 128), (1, 1030, 400, 24, 24, 128)]


@pytest.mark.parametrize("b,l,keys,h,g,d", FORMS)
@pytest.mark.parametrize("scale", [0.002, 0.0625, 1.5])
@pytest.mark.parametrize("first,last", [(128, 0), (200, 60), (0, 0), (10**9, 0)])
def test_masked_blocks(b, l, keys, h, g, d, scale, first, last):
    from tybok_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(l + keys)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=gen).to(torch.bfloat16)  # noqa: E731
    q, k, v = rnd(b * l, h * d), rnd(b, g, keys, d), rnd(b, g, keys, d)
    valid = torch.ones(b, keys, dtype=torch.uint8, device="cuda")
    valid[:, : min(first, keys)] = 0
    if last:
        valid[:, keys - last :] = 0
    call = lambda: ops.attention(q, k, v, valid, tokens=l, keys=keys, scale=scale, out_planes=True)  # noqa: E731
    y, yp = call()
    ops.check_status()
    s = torch.einsum("bthd,bhnd->bhtn", q.view(b, l, h, d).double(), k.double().repeat_interleave(h // g, 1)) * scale
    s = s.masked_fill(valid[:, None, None] == 0, float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)  # no key at all: zero, as the kernels have it
    ref = torch.einsum("bhtn,bhnd->bthd", p, v.double().repeat_interleave(h // g, 1)).reshape(b * l, h * d)
    # probabilities and output are rounded to bf16: 2^-8 of the values' weighted mean magnitude, and of the result
    room = torch.einsum("bhtn,bhnd->bthd", p, v.double().abs().repeat_interleave(h // g, 1)).reshape(b * l, h * d)
    assert bool(((y.double() - ref).abs() <= 2.0**-8 * (room + ref.abs()) + 1e-6).all())
    lib = ops._lib.load()
    trace = torch.zeros(16 * 8192, dtype=torch.int64, device="cuda")
    lib.tybok_debug_set_trace(trace.data_ptr())
    try:
        y1, yp1 = call()
        torch.cuda.synchronize()
    finally:
        lib.tybok_debug_set_trace(None)
    assert torch.equal(y, y1) and torch.equal(yp, yp1)


# Scales that no model uses but the entry takes: zero (the mean of the valid values), below zero, and so small that a finite stand-in for a
# masked score would not be small beside the others.  Keys past the last one count as masked, so the unmasked call is a case too.
@pytest.mark.parametrize("b,l,keys,h,g,d", FORMS)
@pytest.mark.parametrize("scale", [0.0, 1e-30, -0.002, -0.0625])
@pytest.mark.parametrize("first,last", [(0, 0), (128, 37)])
def test_masked_keys_count_for_nothing_at_any_scale(b, l, keys, h, g, d, scale, first, last):
    test_masked_blocks(b, l, keys, h, g, d, scale, min(first, keys // 2), last)


# Two blocks of keys that are merged: one of weight about 2^-130 whose single valid key has values that its weight brings back to order 1.
@pytest.mark.parametrize("b,h,g,keys", [(1, 8, 1, 256), (2, 8, 2, 256), (1, 8, 1, 1024)])  # rows pushed, one more group, staged in L2
def test_a_blocks_small_weight_counts(b, h, g, keys):
    from tybok_b200 import ops

    q = torch.zeros(b * 50, h, 256, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.zeros(b, g, keys, 256, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q[..., 0], k[:, :, 128, 0] = 1.0, -90.0
    v[:, :, 128] = 3e38
    valid = torch.zeros(b, keys, dtype=torch.uint8, device="cuda")
    valid[:, :129] = 1
    y = ops.attention(q.view(b * 50, h * 256), k, v, valid, tokens=50, keys=keys, scale=1.0)[0]
    ops.check_status()
    want = float(torch.exp(torch.tensor(-90.0).double()) * v[0, 0, 128, 0].double() / 128)
    # weight 2^-130 / 128 has 12 bits left; bf16 result
    assert bool(((y.double() - want).abs() <= (2.0**-9 + 2.0**-11) * want).all()), (float(y.min()), float(y.max()), want)
