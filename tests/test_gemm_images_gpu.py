"""The one-tile GEMM's images and its tiles of any token count: where the planes of a token tile are one run of rows, the tile is
the tokens divided by the tiles, and with K over a cluster pairs of rows go round its CTAs.  Each call against a forced tile (a
multiple of 16 tokens, the same K split), whose sums have the same order, and against the image that takes every form (it
runs while the debugging counters are on): the same bits."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu


def _weights(n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return w8_ref.quantize_w8(torch.empty(n, k, device="cuda").normal_(0, 0.02, generator=g))


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


# one token, odd counts, a tile's last row pair half empty, fewer row pairs than CTAs, two tiles of which the second is shorter
@pytest.mark.parametrize("m", [1, 7, 17, 21, 33, 50, 64, 79, 81, 106, 127])
@pytest.mark.parametrize("splits", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("planes", [2, 3])
def test_same_bits_as_a_forced_tile_and_the_general_image(m, splits, planes):
    from tybok_b200 import ops

    n, k = 640, 1152  # a channel tile count that is odd, nine K blocks
    g = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *s: torch.empty(*s, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)  # noqa: E731
    xp, (w8, sc) = ops.split3(rnd(m, k), 4), _weights(n, k, 3)
    res, gate, bias = rnd(m, n), rnd(m, n), rnd(n)
    xp2, rs = ops.norm_planes2(rnd(m, k), ops.NORM_RMS, torch.zeros(k, device="cuda"))
    lin = (lambda **kw: ops.w8x3_linear(xp, 4, w8, sc, **kw)) if planes == 3 else (lambda **kw: ops.w8x2_gemm(xp2, rs, w8, sc, **kw))
    gated = (lambda **kw: ops.w8x3_geglu_packed(xp, 4, w8, sc, **kw)) if planes == 3 else (
        lambda **kw: ops.w8x2_gemm(xp2, rs, w8, sc, epilogue=ops.EPI_GEGLU_PACKED, **kw))
    calls = [lambda t: lin(bias=bias, token_tile=t, splits=splits),
             lambda t: lin(epilogue=ops.EPI_GELU, out_planes=True, token_tile=t, splits=splits),
             lambda t: lin(epilogue=ops.EPI_RESIDUAL, residual=res, gate=gate.float(), rows_per_gate=1, token_tile=t, splits=splits),
             lambda t: gated(out_planes=True, token_tile=t, splits=splits)]
    counters = torch.zeros(16 * 8, dtype=torch.int32, device="cuda")
    lib = ops._lib.load()
    for call in calls:
        y = call(0)
        cap = 64 if planes == 3 else 128
        assert _same(y, call(cap if m > cap else (m + 15) // 16 * 16))
        lib.tybok_debug_set_counters(counters.data_ptr())
        try:
            general = call(0)
            torch.cuda.synchronize()
        finally:
            lib.tybok_debug_set_counters(None)
        assert _same(y, general)
    ops.check_status()
    assert int(counters.sum()) > 0


@pytest.mark.parametrize("m", [1, 5, 16])
def test_few_tokens_in_both_images(m):
    from tybok_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m)
    x, (w8, sc) = torch.empty(m, 2048, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16), _weights(2560, 2048, 5)
    res = torch.empty(m, 2560, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    counters = torch.zeros(16 * 8, dtype=torch.int32, device="cuda")
    lib = ops._lib.load()
    for kw in (dict(), dict(epilogue=ops.EPI_GELU), dict(epilogue=ops.EPI_RESIDUAL, residual=res)):
        y = ops.w8a16_linear(x, w8, sc, **kw)
        lib.tybok_debug_set_counters(counters.data_ptr())
        try:
            general = ops.w8a16_linear(x, w8, sc, **kw)
            torch.cuda.synchronize()
        finally:
            lib.tybok_debug_set_counters(None)
        assert torch.equal(y, general)
    ops.check_status()


# Over 64 tokens in a tile an epilogue warp sends two groups of 16 rows per matrix, in turn: 65 (one row in the second group), odd,
# a full tile, and two tiles of which one is forced.
@pytest.mark.parametrize("m,tile", [(64, 0), (65, 0), (70, 0), (79, 0), (80, 0), (150, 80)])
@pytest.mark.parametrize("splits", [0, 2, 3, 4, 8])
def test_two_matrices_with_k_over_a_cluster(m, tile, splits):
    from tybok_b200 import ops

    i, k = 640, 1024
    g = torch.Generator(device="cuda").manual_seed(m)
    xp = ops.split3(torch.empty(m, k, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16), 4)
    (g8, gs), (u8, us) = _weights(i, k, 3), _weights(i, k, 4)
    two = ops.w8x3_geglu(xp, 4, g8, gs, u8, us, out_planes=True, token_tile=tile, splits=splits)
    one = ops.w8x3_geglu_packed(xp, 4, *ops.pack_gate_up(g8, gs, u8, us), out_planes=True, token_tile=tile, splits=splits)
    ops.check_status()
    assert _same(two, one)
