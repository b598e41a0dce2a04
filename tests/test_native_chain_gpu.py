"""The native chains at the sizes where they branch: token-major keys with and without a partial last block (bit-equal to
one head-major copy), blocks on either side of the two-plane threshold, the batched FFN tail against one call per element."""

import pytest
import torch

from tybok_b200.shapes import DIT_TINY
from tybok_b200.weights import quantize_dit_block, quantize_w8, random_dit_block_params

pytestmark = pytest.mark.gpu


def _rnd(g, *shape, std=1.0):
    return torch.empty(*shape, device="cuda").normal_(0, std, generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("m", [1, 50, 128, 200])
@pytest.mark.parametrize("lv", [1, 127, 128, 129, 300])
def test_token_major_keys_equal_one_head_major_copy(m, lv):
    from tybok_b200 import ops
    from tybok_b200.dit import DiTBlock, DiTDenoiser

    s = DIT_TINY
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + lv)
    params = quantize_dit_block(random_dit_block_params(s, seed=3, device="cuda"))
    den = DiTDenoiser([params], s)
    blk = den.blocks[0]
    a, c = s.heads * s.head_dim, 140
    x, vk, vv, ck, cv = _rnd(g, 1, m, s.hidden), _rnd(g, 1, lv, a), _rnd(g, 1, lv, a), _rnd(g, 1, c, a), _rnd(g, 1, c, a)
    t_mod = _rnd(g, 1, 6, s.hidden, std=0.5)
    freqs = torch.polar(torch.ones(m, s.head_dim // 2, dtype=torch.float64), torch.arange(m, dtype=torch.float64)[:, None] * 0.01
                        + torch.zeros(m, s.head_dim // 2, dtype=torch.float64))[:, None, :].cuda()
    mask = torch.ones(c, dtype=torch.bool)
    mask[-9:-2] = False
    got = den.run_action_layers(x, t_mod, freqs, [{"k": vk, "v": vv}], [(ck, cv)], mask.cuda())
    kc, vc = blk.store_context_kv(vk, vv)
    pad = torch.zeros(1, s.heads, m, s.head_dim, dtype=torch.bfloat16, device="cuda")
    cache = (torch.cat([kc, pad], 2).contiguous(), torch.cat([vc, pad], 2).contiguous())
    f = freqs.reshape(m, -1).to(torch.complex64)
    want = blk.forward(x[0], blk.modulations(t_mod), f.real.float().contiguous(), f.imag.float().contiguous(), cache, lv,
                       blk.store_context_kv(ck, cv), mask[None].to(torch.uint8).cuda())
    ops.check_status()
    assert torch.equal(got[0], want)
    if m == 50:  # an unaligned, non-contiguous caller tensor gives the same
        odd = torch.cat([_rnd(g, 1, lv, 1), vk], dim=2)[:, :, 1:]
        again = den.run_action_layers(x, t_mod, freqs, [{"k": odd, "v": vv}], [(ck, cv)], mask.cuda())
        assert torch.equal(again, got)


@pytest.mark.parametrize("b,s,rows", [(1, 7, "one"), (2, 64, "each"), (3, 43, "mixed"), (2, 515, "each")])
def test_batched_ffn_tail_equals_one_call_per_element(b, s, rows):
    from tybok_b200 import ops
    from tybok_b200.hooks import make_fused_ffn_tail

    h, f = 256, 640
    g = torch.Generator(device="cuda").manual_seed(s)

    class Lin:
        def __init__(self, n, k):
            self.weight, self.weight_scale = quantize_w8(_rnd(g, n, k, std=0.02))
            self.bias = _rnd(g, n)

    class Blk:
        ffn = [Lin(f, h), None, Lin(h, f)]

    fn = make_fused_ffn_tail(Blk)
    x, table = _rnd(g, b, s, h), _rnd(g, b, 6, h, std=0.5)
    mods = [table[:, i : i + 1] for i in (3, 4, 5)]
    if rows == "one":
        mods = [m[0, 0] for m in mods]
    elif rows == "mixed":
        mods[1] = mods[1][:1]
    y = fn(x, *mods)
    ops.check_status()
    assert y.shape == x.shape
    for i in range(b):
        one = [m if m.dim() == 1 else m[min(i, m.shape[0] - 1)] for m in mods]
        ref = fn(x[i], *one)
        assert float((y[i].float() - ref.float()).norm() / ref.float().norm()) <= 2e-3


def _layouts(x):
    """The rows of x [B, L, W] as a host framework may hand them over: with an odd stride, off a 16-byte boundary, both."""
    b, l, w = x.shape
    for wide, off in ((w + 1, 0), (w + 8, 3), (w + 5, 2)):
        t = torch.zeros(b, l, wide, dtype=x.dtype, device=x.device)
        t[:, :, off : off + w] = x
        yield t[:, :, off : off + w]
    yield torch.cat([x.flatten()[:1], x.flatten()])[1:].view(b, l, w)


@pytest.mark.parametrize("m", [1, 5, 70])
def test_hooks_take_rows_of_any_layout(m):
    from tybok_b200 import ops
    from tybok_b200.hooks import make_fused_ffn_tail, make_mlp_forward

    w, f = 256, 640
    g = torch.Generator(device="cuda").manual_seed(m)

    class Lin:
        def __init__(self, n, k):
            self.weight, self.weight_scale = quantize_w8(_rnd(g, n, k, std=0.02))
            self.bias = _rnd(g, n)

    class Mod:
        gate_proj, up_proj, down_proj = Lin(f, w), Lin(f, w), Lin(w, f)
        ffn = [Lin(f, w), None, Lin(w, f)]

    mlp, tail = make_mlp_forward(Mod), make_fused_ffn_tail(Mod)
    x, table = _rnd(g, 2, m, w), _rnd(g, 5, 6, w, std=0.5)
    mods = [table[:2, i : i + 1] for i in (3, 4, 5)]
    want_mlp, want_tail = mlp(x), tail(x, *mods)
    for y in _layouts(x):
        assert torch.equal(mlp(y), want_mlp) and torch.equal(tail(y, *mods), want_tail)
    same = x[:1, :1].expand(2, m, w)  # one row, repeated by a stride of zero
    assert torch.equal(mlp(same), mlp(same.contiguous()))
    assert torch.equal(tail(same, *mods), tail(same.contiguous(), *mods))
    assert torch.equal(tail(x, *(table[:, i : i + 1] for i in (3, 4, 5))), want_tail)  # a table of more rows: the first ones
    ops.check_status()


def test_block_takes_modulation_rows_that_lie_apart():
    from tybok_b200.dit import DiTBlock

    s = DIT_TINY
    g = torch.Generator(device="cuda").manual_seed(2)
    blk = DiTBlock(quantize_dit_block(random_dit_block_params(s, seed=3, device="cuda")), s)
    x, table = _rnd(g, 33, s.hidden), _rnd(g, 6, 2 * s.hidden, std=0.5)
    cos, sin = torch.ones(33, s.head_dim // 2, device="cuda"), torch.zeros(33, s.head_dim // 2, device="cuda")
    cache = lambda: [torch.zeros(1, s.heads, 33, s.head_dim, dtype=torch.bfloat16, device="cuda") for _ in range(2)]  # noqa: E731
    mods = table[:, : s.hidden]
    assert torch.equal(blk.forward(x, mods, cos, sin, cache()), blk.forward(x, mods.contiguous(), cos, sin, cache()))


def test_stack_reserves_what_its_forms_take():
    """Peak of one expert-width layer beside its inputs at batch 32: no exchange workspace where the key loop runs (338 MB), no
    planes of the folded form where the norms are kernels."""
    from tybok_b200 import _lib, ops

    b, w, inner, a, l, keys = 32, 1024, 4096, 2048, 50, 594
    lin = lambda n, k: quantize_w8(torch.full((n, k), 0.01, dtype=torch.bfloat16, device="cuda"))  # noqa: E731
    stack = _lib.native().GemmaStack(w, 8, 1, 256, [(lin(2560, w), lin(w, 2048), lin(2 * inner, w), None, lin(w, inner), None, None)])
    mk = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    mods = [(torch.zeros(1, 3 * w, device="cuda"), torch.zeros(1, 3 * w, device="cuda"))]
    args = (mk(b * l, w), b, l, torch.zeros(b * l, dtype=torch.int32, device="cuda"), mk(700, 256), mk(700, 256), [mk(b, 1, keys, 256)],
            [mk(b, 1, keys, 256)], keys - l, torch.ones(b, keys, dtype=torch.uint8, device="cuda"), mods, None, 0, 1, [], [])
    stack.forward(*args)
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    stack.forward(*args)
    ops.check_status()
    # two planes and a scale of the norm, q, three planes of the attention and of the hidden rows, three bf16 streams, the result
    rows = b * l * (2 * w + 4 + 2 * a + 3 * a + 3 * inner + 3 * 2 * w + 2 * w)
    assert torch.cuda.max_memory_allocated() - base <= rows + (1 << 20)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,n", [(20, 256), (300, 9600)])  # one tile per CTA, which reads gates in vectors; CTA pairs, which do not
def test_gate_off_its_alignment(m, n, dtype):
    from tybok_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(m)
    w8, sc = quantize_w8(_rnd(g, n, 256, std=0.02))
    x, res, gate = _rnd(g, m, 256), _rnd(g, m, n), _rnd(g, 2, n).to(dtype)
    run = lambda gt: ops.w8a16_linear(x, w8, sc, epilogue=ops.EPI_RESIDUAL, residual=res, gate=gt, rows_per_gate=(m + 1) // 2)  # noqa: E731
    want = run(gate)
    for off, wide in ((1, n + 4), (4, n + 3)):
        t = torch.zeros(2 * wide + 8, dtype=dtype, device="cuda")[off : off + 2 * wide].view(2, wide)[:, :n]
        t.copy_(gate)
        if m == 20:
            with pytest.raises(_lib.TybokError, match="gate must be"):
                run(t)
        else:
            assert torch.equal(run(t), want)
    ops.check_status()


# tokens on both sides of the two-plane threshold; interleaved gate / up weights and, at a width that is no multiple of 64, two matrices
@pytest.mark.parametrize("b,l,inner", [(1, 33, 256), (2, 70, 256), (2, 150, 256), (1, 70, 336)])
def test_filling_the_caches_equals_the_whole_pass(b, l, inner):
    """Keys and values of every layer bit for bit, and a stream that waits for a layer's event finds them written."""
    from tybok_b200 import _lib, ops

    w, d, heads, layers = 256, 256, 2, 3
    g = torch.Generator(device="cuda").manual_seed(l)
    lin = lambda n, k: quantize_w8(_rnd(g, n, k, std=0.02))  # noqa: E731
    rows = []
    for _ in range(layers):
        gate, up = lin(inner, w), lin(inner, w)
        ffn = (ops.pack_gate_up(*gate, *up), None) if inner % 64 == 0 else (gate, up)
        norms = [_rnd(g, w, std=0.1).float() for _ in range(2)]
        rows.append((lin((heads + 2) * d, w), lin(w, heads * d), *ffn, lin(w, inner), *norms))
    stack = _lib.native().GemmaStack(w, heads, 1, d, rows)
    x, valid = _rnd(g, b * l, w), torch.ones(b, l, dtype=torch.uint8, device="cuda")
    valid[:, l // 2 : l // 2 + 5] = 0
    pos = torch.arange(l, dtype=torch.int32, device="cuda").repeat(b)
    cos, sin = _rnd(g, l, d), _rnd(g, l, d)
    caches = lambda: ([torch.zeros(b, 1, l + 7, d, dtype=torch.bfloat16, device="cuda") for _ in range(layers)] for _ in range(2))  # noqa: E731
    (kc, vc), (k1, v1) = caches(), caches()
    stack.forward(x, b, l, pos, cos, sin, kc, vc, 0, valid, None, None, 0, layers, [], [])
    done, side = [torch.cuda.Event() for _ in range(layers)], torch.cuda.Stream()
    for ev in done:
        ev.record()
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)  # ten milliseconds in which an event that is not recorded again lets the side stream pass
    stack.fill_caches(x, b, l, pos, cos, sin, k1, v1, valid, [ev.cuda_event for ev in done])
    seen = []
    with torch.cuda.stream(side):
        for i, ev in enumerate(done):
            side.wait_event(ev)
            seen.append((k1[i].clone(), v1[i].clone()))
    torch.cuda.synchronize()
    ops.check_status()
    for i in range(layers):
        assert bool(kc[i][:, :, :l].any()) and not bool(k1[i][:, :, l:].any())
        assert torch.equal(seen[i][0], kc[i]) and torch.equal(seen[i][1], vc[i])
        assert torch.equal(k1[i], kc[i]) and torch.equal(v1[i], vc[i])
