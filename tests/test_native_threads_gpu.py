"""Native calls beside other Python threads: while a call waits for room in the device's launch queue, or returns an error,
the interpreter goes on."""

import threading
import time

import pytest
import torch

from tybok_b200.weights import quantize_w8

pytestmark = pytest.mark.gpu


class _Lin:
    def __init__(self, n, k):
        self.weight, self.weight_scale = quantize_w8(torch.full((n, k), 0.01, dtype=torch.bfloat16, device="cuda"))
        self.bias = torch.zeros(n, dtype=torch.bfloat16, device="cuda")


def _calls():
    from tybok_b200 import _lib, ops
    from tybok_b200.dit import DiTBlock
    from tybok_b200.hooks import make_fused_ffn_tail, make_mlp_forward
    from tybok_b200.shapes import DIT_TINY as s
    from tybok_b200.weights import quantize_dit_block, random_dit_block_params

    bf = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16, device="cuda")  # noqa: E731

    class Mod:
        gate_proj, up_proj, down_proj = _Lin(512, 256), _Lin(512, 256), _Lin(256, 512)
        ffn = [_Lin(512, 256), None, _Lin(256, 512)]

    lin, x, kv = _Lin(256, 256), bf(1, 20, 256), bf(1, 1, 20, 128)
    mlp, tail, mod = make_mlp_forward(Mod), make_fused_ffn_tail(Mod), bf(1, 1, 256)
    blk = DiTBlock(quantize_dit_block(random_dit_block_params(s, seed=0, device="cuda")), s)
    cache = (bf(1, s.heads, 20, s.head_dim), bf(1, s.heads, 20, s.head_dim))
    table = torch.ones(20, s.head_dim // 2, device="cuda")
    w = lambda n, k: quantize_w8(bf(n, k) + 0.01)  # noqa: E731
    norm, q, kc, vc = torch.zeros(256, device="cuda"), bf(20, 128), kv.clone(), kv.clone()
    bx, mods = bf(20, s.hidden), bf(6, s.hidden)
    stack = _lib.native().GemmaStack(256, 2, 1, 128, [(w(512, 256), w(256, 256), w(1024, 256), None, w(256, 512), norm, norm)])
    pos, rope, valid = torch.zeros(20, dtype=torch.int32, device="cuda"), bf(32, 128), torch.ones(1, 20, dtype=torch.uint8, device="cuda")
    return {
        "linear": lambda: ops.w8a16_linear(x, lin.weight, lin.weight_scale, lin.bias),
        "attention": lambda: ops.attention(q, kv, kv, tokens=20, keys=20, scale=1.0),
        "mlp": lambda: mlp(x),
        "ffn_tail": lambda: tail(x, mod, mod, mod),
        "dit_block": lambda: blk.forward(bx, mods, table, table, cache),
        "gemma_stack": lambda: stack.forward(x[0], 1, 20, pos, rope, rope, [kc], [vc], 0, valid, None, None, 0, 1, [], []),
    }


def _longest_stall(call):
    """Seconds that a ticking thread stood still while ``call`` ran into a launch queue filled behind a sleeping device."""
    stop, longest = threading.Event(), [0.0]

    def ticker():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            longest[0] = max(longest[0], now - last)
            last = now

    thread = threading.Thread(target=ticker)
    thread.start()
    try:
        t0 = time.perf_counter()
        torch.cuda._sleep(1_000_000_000)  # half a second of device time, behind which the queue fills
        while time.perf_counter() - t0 < 0.25:
            call()
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    return longest[0]


@pytest.mark.parametrize("name", ["linear", "attention", "mlp", "ffn_tail", "dit_block", "gemma_stack"])
def test_other_threads_run_while_a_call_waits_for_the_launch_queue(name):
    call = _calls()[name]
    for _ in range(3):
        call()
    torch.cuda.synchronize()
    # a call that holds the lock stalls the others every time; a busy host may do so once
    assert min(_longest_stall(call) for _ in range(3)) < 0.1


def test_errors_of_calls_without_the_lock():
    from tybok_b200 import _lib, ops

    lin = _Lin(256, 256)
    kv = torch.zeros(1, 1, 20, 128, dtype=torch.bfloat16, device="cuda")
    for _ in range(3):
        with pytest.raises(_lib.TybokError, match="Lk <= Lcap"):
            ops.attention(torch.zeros(4, 128, dtype=torch.bfloat16, device="cuda"), kv, kv, tokens=4, keys=21, scale=1.0)
        with pytest.raises(TypeError, match="must be bf16"):
            ops.w8a16_linear(torch.zeros(4, 256, device="cuda"), lin.weight, lin.weight_scale)
        with pytest.raises(ValueError, match="planes have K"):
            ops.w8a16_linear(kv[0, 0], lin.weight, lin.weight_scale)
        with pytest.raises(NotImplementedError, match="no CPU implementation"):
            ops.attention(kv[0, 0].cpu(), kv.cpu(), kv.cpu(), tokens=20, keys=20, scale=1.0)
    ops.check_status()
