"""The block-scaled two-plane form: ``x * 2**k = e4m3 + e5m2`` with one k per token and 32 channels, and the CTA-pair GEMM whose
MMA applies the scales.  Planes against a restatement of the split in float64; the GEMM at the edges of its tiles against the
float64 product of what the planes hold, every epilogue, K whole and over a cluster; the hooks and the linear at sizes that
take the form, against the oracle; a wait that runs out."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu


def _lib():
    from tybok_b200 import ops

    return ops._lib, ops._lib.load(), torch.cuda.current_stream().cuda_stream


def _x(m, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=g)  # noqa: E731
    return (n(m, k) * torch.exp(2 * n(m, 1)) * torch.exp(n(1, k))).to(torch.bfloat16)  # rows and channels of other magnitudes


def _weights(n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return w8_ref.quantize_w8(torch.empty(n, k, device="cuda").normal_(0, 0.02, generator=g))


def _split(x):
    mod, lib, st = _lib()
    m, k = x.shape
    planes = torch.empty(2, m, k, dtype=torch.uint8, device="cuda")
    sf = torch.empty(k // 128, m, dtype=torch.int32, device="cuda")
    mod.check(lib.tybok_split_mx(x.data_ptr(), x.stride(0), planes.data_ptr(), sf.data_ptr(), m, k, st), "split")
    return planes, sf


def _scales(sf, m, k):
    return sf.view(torch.uint8).reshape(k // 128, m, 4).permute(1, 0, 2).reshape(m, k // 32)


def _values(planes, sf):
    _, m, k = planes.shape
    both = planes[0].view(torch.float8_e4m3fn).double() + planes[1].view(torch.float8_e5m2).double()
    return both * torch.exp2(_scales(sf, m, k).double() - 127).repeat_interleave(32, 1)


def _gemm(planes, sf, w8, sc, bias=None, epi=0, res=None, gate=None, rows=1, out_planes=False, splits=0):
    from tybok_b200 import ops

    mod, lib, st = _lib()
    (n, k), m = w8.shape, planes.shape[1]
    n_out = n // 2 if epi == 4 else n
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    y = torch.empty(m, n_out, dtype=torch.bfloat16, device="cuda")
    yp = torch.empty(2, m, n_out, dtype=torch.uint8, device="cuda") if out_planes else None
    ys = torch.empty(n_out // 128, m, dtype=torch.int32, device="cuda") if out_planes else None
    mod.check(lib.tybok_w8mx_gemm(p(planes), p(sf), None, p(w8), p(sc), p(bias), p(y), n_out, p(yp), p(ys), m, n, k, epi, p(res), n,
                                  p(gate), n, rows, int(gate is not None and gate.dtype == torch.bfloat16), splits,
                                  p(ops.status_word(planes.device)), st), "gemm")
    ops.check_status()
    return y, yp, ys


def _check_planes(x, planes, sf):
    """Exact where |x'| >= 2^-6, off by at most 2^-14 scaled units below; the block maximum lands in (224, 448]."""
    m, k = x.shape
    scale = torch.exp2(_scales(sf, m, k).double() - 127).repeat_interleave(32, 1)
    got, want = _values(planes, sf) / scale, x.double() / scale
    big = want.abs() >= 2.0**-6
    assert torch.equal(got[big], want[big])
    assert float((got - want).abs().max()) <= 2.0**-14
    top = want.abs().reshape(m, -1, 32).amax(2)
    assert bool(((top > 224) & (top <= 448) | (top < 2.0**-100)).all())


@pytest.mark.parametrize("m,k", [(1, 128), (7, 384), (333, 2048), (129, 14336)])
def test_split(m, k):
    x = _x(m, k, m)
    x[0, :32] = 0
    x[m - 1, 32:64] = 1e-30  # below any activation, still a normal bf16 block
    x[m // 2, 64:96] *= 1e20
    _check_planes(x, *_split(x))


def test_split_keeps_what_is_not_finite():
    x = _x(4, 256, 1)
    x[1, 40], x[2, 200] = float("inf"), float("nan")
    planes, sf = _split(x)
    s = _scales(sf, 4, 256)
    assert s[1, 1] == 255 and s[2, 6] == 255 and int((s == 255).sum()) == 2  # UE8M0 NaN: the whole row of the product
    y, _, _ = _gemm(planes, sf, *_weights(256, 256, 2))
    assert bool(y[1].isnan().all() and y[2].isnan().all() and y[0].isfinite().all() and y[3].isfinite().all())


# token tiles of one and two sizes up to 240, half-filled last chunks, channel tiles cut at 128 and 4, one K block, batches of
# four K blocks with a rest, several tiles per pair, K over two to four pairs
@pytest.mark.parametrize("m,n,k,splits", [(1, 256, 128, 1), (16, 384, 640, 1), (129, 260, 384, 1), (241, 19072, 512, 1), (257, 6400, 1152, 1),
                                          (1000, 3332, 640, 1), (4111, 1028, 256, 1), (333, 2048, 4096, 2), (200, 516, 2176, 2), (50, 256, 16384, 2)])
def test_gemm_at_tile_edges(m, n, k, splits):
    x, (w8, sc) = _x(m, k, m + n), _weights(n, k, n)
    planes, sf = _split(x)
    values, w = _values(planes, sf), w8.double()
    prod = (values @ w.T) * sc.double()
    slack = (values.abs() @ w.abs().T) * sc.double() * 2.0**-20  # fp32 accumulation
    g = torch.Generator(device="cuda").manual_seed(3)
    bias = torch.empty(n, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    res = torch.empty(m, n, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    rows = (m + 2) // 3
    gate = torch.empty(3, n, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    lin = prod + bias.double()
    gated = lin * gate.double().repeat_interleave(rows, 0)[:m]

    def close(y, want, extra):  # the last rounding to bf16 (8 significant bits) is off by 2^-8 of its value at most
        assert bool(((y.double() - want).abs() <= 1.01 * 2.0**-8 * want.abs() + extra).all())

    close(_gemm(planes, sf, w8, sc, splits=splits)[0], prod, slack)
    y, yp, ys = _gemm(planes, sf, w8, sc, bias, epi=1, out_planes=n % 128 == 0, splits=splits)
    close(y, torch.nn.functional.gelu(lin, approximate="tanh"), 1.2 * (slack + 2.0**-8 * lin.abs()) + 1e-6)  # |gelu'| < 1.13
    if yp is not None:
        _check_planes(y, yp, ys)
    y = _gemm(planes, sf, w8, sc, bias, epi=2, res=res, gate=gate, rows=rows, splits=splits)[0]
    close(y, res.double() + gated, 2.02 * 2.0**-8 * gated.abs() + 1.1 * slack * gate.double().abs().repeat_interleave(rows, 0)[:m])
    assert torch.equal(y, _gemm(planes, sf, w8, sc, bias, epi=2, res=res, gate=gate, rows=rows, splits=splits)[0])


@pytest.mark.parametrize("m,i,k", [(300, 512, 256), (544, 4096, 512), (113, 9472, 128)])
def test_gated_form_and_its_planes(m, i, k):
    from tybok_b200 import ops

    gate, up, x = _weights(i, k, 1), _weights(i, k, 2), _x(m, k, 3) * 0.1
    w8, sc = ops.pack_gate_up(*gate, *up)
    ref = w8_ref.gelu_tanh(w8_ref.w8_linear(x.cpu(), gate[0].cpu(), gate[1].cpu())) * w8_ref.w8_linear(x.cpu(), up[0].cpu(), up[1].cpu())
    planes, sf = _split(x)
    y, yp, ys = _gemm(planes, sf, w8, sc, epi=4, out_planes=True)
    assert w8_ref.rel_l2(y.cpu(), ref) <= 1e-2
    _check_planes(y, yp, ys)


@pytest.mark.parametrize("m,w,groups", [(1, 128, 1), (129, 1024, 1), (300, 2048, 2), (1000, 3072, 5), (65, 4096, 1)])
def test_layernorm_into_the_form(m, w, groups):
    """Against the row kernel's bf16 rows: the sums run in another order, so a rounding may fall the other way."""
    from tybok_b200 import ops

    mod, lib, st = _lib()
    x = _x(m, w, w)
    g = torch.Generator(device="cuda").manual_seed(4)
    sh, sc = (torch.empty(groups, w, device="cuda").normal_(0, 0.5, generator=g).to(torch.bfloat16) for _ in range(2))
    per = -(-m // groups)
    planes = torch.empty(2, m, w, dtype=torch.uint8, device="cuda")
    sf = torch.empty(w // 128, m, dtype=torch.int32, device="cuda")
    mod.check(lib.tybok_layernorm_modulate_mx(x.data_ptr(), w, sh.data_ptr(), sc.data_ptr(), w, per, m, w, 1e-6, planes.data_ptr(),
                                              sf.data_ptr(), st), "ln")
    ref = torch.cat([ops.layernorm_modulate(x[i * per : (i + 1) * per], sh[i], sc[i], out_bf16=True, out_planes=False)[0]
                     for i in range(groups) if i * per < m])
    got = _values(planes, sf)
    assert torch.equal(got.to(torch.bfloat16).double(), got) or float((got - got.to(torch.bfloat16).double()).abs().max()) <= 1e-6 * float(got.abs().max())
    # three roundings of values up to (|LN| + 1) * (1 + |scale|) + |shift|, each off by one ulp at most
    room = 2.0**-7 * (ref.double().abs() + sh.double().abs().repeat_interleave(per, 0)[:m] + 1e-3)
    assert bool(((got - ref.double()).abs() <= 3 * room).all()) and w8_ref.rel_l2(got.float(), ref.float()) <= 1e-3


def test_which_products_take_the_form():
    _, lib, _ = _lib()
    assert lib.tybok_w8mx_suits(4146, 14336, 3072) and lib.tybok_w8mx_suits(333, 2048, 16384)
    for m, n, k in [(160, 16384, 2048), (50, 8192, 1024), (800, 2560, 1024), (4146, 14336, 3080), (4146, 14336, 0)]:
        assert not lib.tybok_w8mx_suits(m, n, k)


@pytest.mark.parametrize("m,n,k,epi", [(333, 2048, 16384, 2), (301, 16384, 2048, 1), (801, 16384, 2048, 0)])
def test_linear_takes_it_and_matches_the_oracle(m, n, k, epi):
    from tybok_b200 import ops

    _, lib, _ = _lib()
    assert lib.tybok_w8mx_suits(m, n, k)
    g = torch.Generator().manual_seed(m)
    x, (w8, sc) = torch.empty(m, k).normal_(0, 1, generator=g).to(torch.bfloat16), _weights(n, k, 7)
    wide = torch.zeros(m, k + 64, dtype=torch.bfloat16, device="cuda")  # a strided view of wider rows
    wide[:, :k] = x.cuda()
    res = torch.empty(m, n).normal_(0, 1, generator=g).to(torch.bfloat16)
    y = ops.w8a16_linear(wide[:, :k], w8, sc, epilogue=epi, residual=res.cuda() if epi == 2 else None)
    ops.check_status()
    lin = w8_ref.w8_linear(x, w8.cpu(), sc.cpu())
    assert w8_ref.rel_l2(y.cpu(), {0: lin, 1: w8_ref.gelu_tanh(lin), 2: res + lin}[epi]) <= 1e-2
    # three planes on the same rows: fp32 summation order only
    y3 = ops.w8a16_linear(wide[:, :k], w8, sc, epilogue=epi, residual=res.cuda() if epi == 2 else None, token_tile=64, splits=1)
    assert w8_ref.rel_l2(y.float(), y3.float()) <= 1e-3


def test_hooks_take_it_and_match_the_oracle():
    from tybok_b200 import hooks

    class M:
        pass

    def lin(n, k, bias, seed):
        m = M()
        (m.weight, m.weight_scale) = _weights(n, k, seed)
        m.bias = torch.randn(n, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda() * 0.1 if bias else None
        return m

    cpu = lambda m: (m.weight.cpu(), m.weight_scale.cpu())  # noqa: E731
    g = torch.Generator().manual_seed(9)
    mlp = M()
    mlp.gate_proj, mlp.up_proj, mlp.down_proj = lin(16384, 2048, False, 1), lin(16384, 2048, False, 2), lin(2048, 16384, False, 3)
    x = torch.randn(1, 345, 2048, generator=g).to(torch.bfloat16)
    ref = w8_ref.gemma_mlp(x, cpu(mlp.gate_proj), cpu(mlp.up_proj), cpu(mlp.down_proj))
    assert w8_ref.rel_l2(hooks.make_mlp_forward(mlp)(x.cuda()).cpu(), ref) <= 1e-2
    blk = M()
    blk.ffn = [lin(14336, 3072, True, 4), None, lin(3072, 14336, True, 5)]
    x = torch.randn(2, 201, 3072, generator=g).to(torch.bfloat16)
    mods = (torch.randn(2, 6, 3072, generator=g) * 0.5).to(torch.bfloat16)
    ref = w8_ref.dit_ffn_tail(x, *(mods[:, i : i + 1] for i in (3, 4, 5)), (*cpu(blk.ffn[0]), blk.ffn[0].bias.cpu()),
                              (*cpu(blk.ffn[2]), blk.ffn[2].bias.cpu()))
    cm = mods.cuda()
    y = hooks.make_fused_ffn_tail(blk)(x.cuda(), *(cm[:, i : i + 1] for i in (3, 4, 5)))
    assert w8_ref.rel_l2(y.cpu().float() - x.float(), ref.float() - x.float()) <= 1e-2


@pytest.mark.parametrize("m,n,k,splits", [(300, 19072, 256, 1), (700, 9600, 4096, 1), (333, 2048, 16384, 2)])
def test_a_wait_that_runs_out(m, n, k, splits):
    from tybok_b200 import ops

    _, lib, _ = _lib()
    w, (planes, sf) = _weights(n, k, 0), _split(_x(m, k, 0))
    good = _gemm(planes, sf, *w, splits=splits)[0]
    lib.tybok_debug_set_epilogue_wait_limit(1)
    try:
        with pytest.raises(ops._lib.TybokError, match="bounded wait"):
            _gemm(planes, sf, *w, splits=splits)
    finally:
        lib.tybok_debug_set_epilogue_wait_limit(0)
    assert torch.equal(_gemm(planes, sf, *w, splits=splits)[0], good)


def test_what_is_refused():
    _, lib, st = _lib()
    x = torch.zeros(4, 512, dtype=torch.bfloat16, device="cuda")
    b = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda").data_ptr()
    f = torch.zeros(1 << 12, device="cuda").data_ptr()
    assert lib.tybok_split_mx(x.data_ptr(), 512, b, b, 4, 200, st) == 1 and lib.tybok_split_mx(x.data_ptr() + 2, 512, b, b, 4, 256, st) == 1
    gemm = lambda sf, rs, yp, ys, n, k, epi: lib.tybok_w8mx_gemm(b, sf, rs, b, f, None, b, n, yp, ys, 4, n, k, epi, b, n, None, 0, 1, 0, 0, None, st)  # noqa: E731
    for call in [(b, f, None, None, 256, 256, 0), (None, None, None, None, 256, 256, 0), (b, None, b, None, 256, 256, 0), (b, None, None, None, 256, 144, 0),
                 (b, None, b, b, 260, 256, 0), (b, None, b, b, 256, 256, 2), (b, None, None, None, 256, 256, 5), (b + 2, None, None, None, 256, 256, 0)]:
        assert gemm(*call) == 1
