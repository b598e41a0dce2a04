"""The one-launch form for up to 16 tokens (the GEMM makes its activation planes itself) is bit-equal to planes plus GEMM:
token counts up to the limit and past it, K tails, more K blocks than ring stages, strided rows, every epilogue."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 16, 17])
@pytest.mark.parametrize("n,k", [(2560, 2048), (128, 272), (132, 16384), (16384, 2048), (18944, 144), (18948, 144)])
def test_linear(m, n, k):
    from tybok_b200 import ops

    g = torch.Generator().manual_seed(m + n)
    w8, sc = (t.cuda() for t in w8_ref.quantize_w8(torch.empty(n, k).normal_(0, 0.02, generator=g)))
    rnd = lambda *s: torch.empty(*s).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()  # noqa: E731
    x = rnd(m, k + 8)[:, :k]  # rows with a stride
    bias, res, gate = rnd(n), rnd(m, n), rnd(1, n)
    for kw in (dict(), dict(epilogue=ops.EPI_GELU), dict(epilogue=ops.EPI_RESIDUAL, residual=res, gate=gate, rows_per_gate=m)):
        y = ops.w8a16_linear(x, w8, sc, bias, **kw)
        ref, _ = ops.w8x3_linear(ops.split3(x, 4), 4, w8, sc, bias, **kw)
        ops.check_status()
        assert torch.equal(y, ref)


@pytest.mark.parametrize("m,w,i", [(1, 1024, 4096), (16, 256, 576), (5, 2048, 16384)])
def test_mlp_hook(m, w, i):
    from tybok_b200 import ops
    from tybok_b200.hooks import make_mlp_forward

    g = torch.Generator(device="cuda").manual_seed(m)

    class Lin:
        def __init__(self, n, k):
            self.weight, self.weight_scale = w8_ref.quantize_w8(torch.empty(n, k, device="cuda").normal_(0, 0.02, generator=g))

    class Mlp:
        gate_proj, up_proj, down_proj = Lin(i, w), Lin(i, w), Lin(w, i)

    x = torch.empty(1, m, w, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    y = make_mlp_forward(Mlp)(x)
    pairs = [(l.weight, l.weight_scale) for l in (Mlp.gate_proj, Mlp.up_proj, Mlp.down_proj)]
    _, hp = ops.w8x3_geglu_packed(ops.split3(x[0], 4), 4, *ops.pack_gate_up(*pairs[0], *pairs[1]), out_bf16=False, out_planes=True)
    ref, _ = ops.w8x3_linear(hp, 4, *pairs[2])
    ops.check_status()
    assert torch.equal(y[0], ref)
