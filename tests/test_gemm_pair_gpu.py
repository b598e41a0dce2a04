"""The persistent CTA-pair GEMM (many output tiles) at the edges of its tiles: token counts around the 32-token steps
and the accumulator widths, channel counts that leave part of a 256- or 512-row tile empty, K tails, few and many tiles
per pair; every epilogue, both activation forms.  Each case against the one-tile-per-CTA kernel (forced token tile and
split) on the same operands, and plain ones against the oracle."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu


def _weights(n, k, seed):
    g = torch.Generator().manual_seed(seed)
    w8, scale = w8_ref.quantize_w8(torch.empty(n, k).normal_(0, 0.02, generator=g))
    return w8.cuda(), scale.cuda()


def _x(m, k, seed):
    return torch.empty(m, k).normal_(0, 1, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16)


@pytest.mark.parametrize("planes", [2, 3])
@pytest.mark.parametrize("m,n,k", [(1, 19072, 144), (81, 9600, 256), (128, 19204, 128), (129, 9476, 400), (257, 6400, 272),
                                   (289, 7172, 128), (1000, 3332, 640), (4111, 1028, 256)])
def test_linear_at_tile_edges(m, n, k, planes):
    from tybok_b200 import ops

    x, (w8, sc) = _x(m, k, m + n), _weights(n, k, n)
    if planes == 3:
        xp = ops.split3(x.cuda(), 4)
        run = lambda **kw: ops.w8x3_linear(xp, 4, w8, sc, **kw)  # noqa: E731
        ref_x = x
    else:
        xp, rs = ops.norm_planes2(x.cuda(), ops.NORM_RMS, torch.zeros(k, device="cuda"))
        run = lambda **kw: ops.w8x2_gemm(xp, rs, w8, sc, **kw)  # noqa: E731
        ref_x = ops.rmsnorm(x.cuda(), weight=torch.zeros(k, device="cuda"), out_bf16=True)[0].cpu()
    g = torch.Generator().manual_seed(5)
    res = torch.empty(m, n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    rows = (m + 2) // 3  # three gate groups, so that tiles straddle them
    gate = torch.empty(3, n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    bias = torch.empty(n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    forms = [dict(), dict(bias=bias, epilogue=ops.EPI_GELU, out_planes=True),
             dict(bias=bias, epilogue=ops.EPI_RESIDUAL, residual=res, gate=gate, rows_per_gate=rows),
             dict(epilogue=ops.EPI_RESIDUAL, residual=res, gate=gate[:1].float(), rows_per_gate=m, out_planes=True)]
    for kw in forms:
        y, yp = run(**kw)
        y1, yp1 = run(token_tile=64, splits=1, **kw)
        ops.check_status()
        if m <= 128:
            assert torch.equal(y, y1) and torch.equal(yp, yp1)  # same order of summation
        assert w8_ref.rel_l2(y.float().cpu(), y1.float().cpu()) <= 2e-3
        if kw.get("out_planes"):
            f = lambda p: p.view(torch.float8_e5m2).float().sum(0)  # noqa: E731
            assert w8_ref.rel_l2(f(yp).cpu(), f(yp1).cpu()) <= 2e-3
    assert w8_ref.rel_l2(run()[0].cpu(), w8_ref.w8_linear(ref_x, w8.cpu(), sc.cpu())) <= 1e-2


@pytest.mark.parametrize("m,i,k", [(3, 9536, 128), (97, 4800, 272), (131, 4736, 128), (545, 1600, 256), (2100, 448, 144)])
def test_gated_form_at_tile_edges(m, i, k):
    from tybok_b200 import ops

    (g8, gs), (u8, us) = _weights(i, k, 1), _weights(i, k, 2)
    p8, ps = ops.pack_gate_up(g8, gs, u8, us)
    x = _x(m, k, m)
    xp = ops.split3(x.cuda(), 4)
    h0, hp0 = ops.w8x3_geglu(xp, 4, g8, gs, u8, us, out_planes=True)
    h1, hp1 = ops.w8x3_geglu_packed(xp, 4, p8, ps, out_planes=True)
    h2, _ = ops.w8x3_geglu_packed(xp, 4, p8, ps, token_tile=64, splits=1)
    ops.check_status()
    assert torch.equal(h0, h1) and torch.equal(hp0, hp1)
    assert w8_ref.rel_l2(h1.cpu(), h2.cpu()) <= 2e-3


@pytest.mark.parametrize("b,l,h,gr,d,key_off", [(1, 1100, 8, 1, 256, 0), (3, 707, 3, 1, 256, 7), (2, 830, 8, 2, 128, 1)])
def test_rotary_form_at_tile_edges(b, l, h, gr, d, key_off):
    from tybok_b200 import ops

    k = 272
    w8, sc = _weights((h + 2 * gr) * d, k, 9)
    wp, sp = ops.pair_qkv_rows(w8, sc, d)
    xp = ops.split3(_x(b * l, k, l).cuda(), 4)
    pos = (torch.arange(l, dtype=torch.int32)[None] + torch.arange(b, dtype=torch.int32)[:, None] * 3).reshape(-1).cuda()
    cos, sin = w8_ref.rope_cos_sin(torch.arange(l + 16)[None], d, torch.bfloat16)
    cos, sin = cos[0].contiguous().cuda(), sin[0].contiguous().cuda()
    c = [torch.zeros(b, gr, key_off + l + 3, d, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    q0 = ops.w8x3_qkv_rope(xp, 4, wp, sp, pos, cos, sin, c[0], c[1], heads=h, key_off=key_off)
    q1 = ops.w8x3_qkv_rope(xp, 4, wp, sp, pos, cos, sin, c[2], c[3], heads=h, key_off=key_off, token_tile=64, splits=1)
    ops.check_status()
    for a, r in ((q0, q1), (c[0], c[2]), (c[1], c[3])):
        assert w8_ref.rel_l2(a.float().cpu(), r.float().cpu()) <= 2e-3
    assert not c[0][:, :, :key_off].any() and not c[0][:, :, key_off + l :].any()


@pytest.mark.parametrize("m,n,k", [(333, 2048, 16384), (257, 2044, 16400), (512, 1796, 12304), (200, 3072, 14336)])
def test_k_split_over_the_pairs_of_a_cluster(m, n, k):
    """Long K with a tile count that fills neither kernel's plain plan: parts exchanged through shared memory, every
    epilogue, two launches bit-equal."""
    from tybok_b200 import ops

    x, (w8, sc) = _x(m, k, m), _weights(n, k, n)
    xp = ops.split3(x.cuda(), 4)
    g = torch.Generator().manual_seed(7)
    res = torch.empty(m, n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    gate = torch.empty(2, n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    bias = torch.empty(n).normal_(0, 1, generator=g).to(torch.bfloat16).cuda()
    for kw in (dict(), dict(bias=bias, epilogue=ops.EPI_GELU, out_planes=True),
               dict(bias=bias, epilogue=ops.EPI_RESIDUAL, residual=res, gate=gate, rows_per_gate=(m + 1) // 2)):
        y, yp = ops.w8x3_linear(xp, 4, w8, sc, **kw)
        again, _ = ops.w8x3_linear(xp, 4, w8, sc, **kw)
        y1, yp1 = ops.w8x3_linear(xp, 4, w8, sc, token_tile=64, splits=1, **kw)
        ops.check_status()
        assert torch.equal(y, again)
        assert w8_ref.rel_l2(y.float().cpu(), y1.float().cpu()) <= 2e-3
        if kw.get("out_planes"):
            f = lambda p: p.view(torch.float8_e5m2).float().sum(0)  # noqa: E731
            assert w8_ref.rel_l2(f(yp).cpu(), f(yp1).cpu()) <= 2e-3
    assert w8_ref.rel_l2(ops.w8x3_linear(xp, 4, w8, sc)[0].cpu(), w8_ref.w8_linear(x, w8.cpu(), sc.cpu())) <= 1e-2
