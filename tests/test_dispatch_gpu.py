"""The calls that go straight to the native extension are still torch ops to whoever intercepts those: ``vmap`` runs them
slice by slice, a dispatch mode sees them by name, a subclass comes back as one."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from tybok_b200.weights import quantize_w8

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore:There is a performance drop")]


class _Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


class _Sub(torch.Tensor):
    pass


def _calls():
    from tybok_b200 import ops
    from tybok_b200.hooks import make_fused_ffn_tail, make_mlp_forward

    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)  # noqa: E731

    class Lin:
        def __init__(self, n, k):
            self.weight, self.weight_scale = quantize_w8(rnd(n, k) * 0.02)
            self.bias = rnd(n)

    class Mod:
        gate_proj, up_proj, down_proj = Lin(512, 256), Lin(512, 256), Lin(256, 512)
        ffn = [Lin(512, 256), None, Lin(256, 512)]

    lin, kv, mlp, tail = Lin(512, 256), rnd(1, 1, 20, 256), make_mlp_forward(Mod), make_fused_ffn_tail(Mod)
    mods = [rnd(1, 1, 256) for _ in range(3)]
    return rnd(3, 20, 256), {
        "w8a16_linear": lambda x: ops.w8a16_linear(x, lin.weight, lin.weight_scale, lin.bias),
        "attention": lambda x: ops.attention(x, kv, kv, tokens=20, keys=20, scale=0.1)[0],
        "mlp": mlp,
        "ffn_tail": lambda x: tail(x, *mods),
    }


@pytest.mark.parametrize("name", ["w8a16_linear", "attention", "mlp", "ffn_tail"])
def test_interception(name):
    xs, calls = _calls()
    call = calls[name]
    want = torch.stack([call(x) for x in xs])
    assert torch.equal(torch.vmap(call)(xs), want)
    with _Seen() as seen:
        y = call(xs[1].clone())
    assert f"tybok_b200.{name}.default" in seen.names and torch.equal(y, want[1])
    z = call(xs[2].as_subclass(_Sub))
    assert type(z) is _Sub and torch.equal(z.as_subclass(torch.Tensor), want[2])
    assert torch.equal(call(torch.nn.Parameter(xs[0], requires_grad=False)), want[0])
