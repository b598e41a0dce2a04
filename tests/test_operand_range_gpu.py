"""Activations beside much larger ones keep all their bits: in every call that makes its own planes, one channel of each 32 is large
and meets zero weights, so the result shows the operand error of its neighbours alone.  Against float64 with the modules' bf16
rounding points; at token counts on both sides of the change from one tile per CTA to a CTA pair."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu

STEP = 2.0**-9  # rounding to bf16 moves a value by this share of it at most


def _bf(x):
    return x.to(torch.bfloat16).double()


def _normal(seed, *shape, std=1.0):
    return torch.empty(*shape, device="cuda").normal_(0, std, generator=torch.Generator(device="cuda").manual_seed(seed))


def _linear(n, k, seed, large_rows=None, zero_columns=False):
    w = _normal(seed, n, k, std=0.02)
    if large_rows is not None:
        w *= large_rows[0]
        w[5::32] *= large_rows[1] / large_rows[0]
    if zero_columns:
        w[:, 5::32] = 0
    m = torch.nn.Module()
    m.weight, m.weight_scale = w8_ref.quantize_w8(w)
    m.bias = None
    return m, m.weight.double() * m.weight_scale.double()[:, None]


@pytest.mark.parametrize("m,n,k", [(100, 2048, 2048), (161, 16384, 2048), (333, 2048, 16384), (801, 16384, 2048)])
def test_linear(m, n, k):
    from tybok_b200 import ops

    x = _normal(m, m, k, std=0.01).to(torch.bfloat16)
    x[:, 5::32] = 1000
    lin, w = _linear(n, k, 1, zero_columns=True)
    y = ops.w8a16_linear(x, lin.weight, lin.weight_scale)
    ops.check_status()
    # the result's rounding; below 4.9e-4 three planes are off by up to 5e-7, a 2e-5th of the values here
    assert w8_ref.rel_l2(y.double(), x.double() @ w.T) <= STEP + 2e-5


@pytest.mark.parametrize("m", [100, 345, 900])
def test_mlp_hook(m):
    from tybok_b200 import hooks

    mlp = torch.nn.Module()
    mlp.gate_proj, wg = _linear(16384, 2048, 1)
    mlp.up_proj, wu = _linear(16384, 2048, 2, large_rows=(0.0005, 200.0))
    mlp.down_proj, wd = _linear(2048, 16384, 3, zero_columns=True)
    x = _normal(m, 1, m, 2048).to(torch.bfloat16)
    y = hooks.make_mlp_forward(mlp)(x)
    xd = x[0].double()
    act = _bf(torch.nn.functional.gelu(_bf(xd @ wg.T), approximate="tanh"))
    ref = _bf(act * _bf(xd @ wu.T)) @ wd.T
    # the result's rounding; GELU and product one bf16 step off at most; 5e-7 of plane error beside hidden values of 4e-4
    assert w8_ref.rel_l2(y[0].double(), ref) <= STEP + 4 * STEP + 1.3e-3


@pytest.mark.parametrize("m", [100, 201, 1000])
def test_ffn_tail_hook(m):
    from tybok_b200 import hooks

    h, f = 3072, 14336
    blk = torch.nn.Module()
    up, wu = _linear(f, h, 1, zero_columns=True)
    down, wd = _linear(h, f, 2)
    up.bias, down.bias = (torch.zeros(n, device="cuda", dtype=torch.bfloat16) for n in (f, h))
    blk.ffn = [up, None, down]
    x = _normal(m, 1, m, h).to(torch.bfloat16)
    scale = torch.full((1, 1, h), 2.0**-8 - 1, device="cuda", dtype=torch.bfloat16)
    scale[..., 5::32] = 1000
    shift, gate = torch.zeros_like(scale), torch.full_like(scale, 1024.0)
    y = hooks.make_fused_ffn_tail(blk)(x, shift, scale, gate)
    xd = x[0].double()
    n = _bf((xd - xd.mean(-1, keepdim=True)) * torch.rsqrt(xd.var(-1, unbiased=False, keepdim=True) + 1e-6))
    hid = _bf(torch.nn.functional.gelu(_bf(_bf(n * _bf(1 + scale[0].double())) @ wu.T), approximate="tanh"))
    ref = xd + 1024.0 * (hid @ wd.T)
    # roundings of the linear and of the sum; pre-activation and GELU one bf16 step off at most; 5e-7 of plane error beside 4e-3
    assert w8_ref.rel_l2(y[0].double(), ref) <= 2 * STEP + 4 * STEP + 2e-4
