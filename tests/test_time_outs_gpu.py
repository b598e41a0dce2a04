"""Every kernel with bounded waits comes back when one runs out: the epilogue's or softmax warps' limit is set to one SM
clock, which no accumulator meets, the launch reports it in the status word, and the next launch gives the same bits as
before.  What runs on the device is the kernels' own unwinding: copies and products in flight are seen to their end, tensor
memory is freed, the CTAs leave."""

import pytest
import torch

from oracle import w8_ref

pytestmark = pytest.mark.gpu

CONVERT, EPILOGUE = 103, 104  # TYBOK_DEV_TIMEOUT_*


def _weights(n, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return w8_ref.quantize_w8(torch.empty(n, k, device="cuda").normal_(0, 0.02, generator=g))


def _x(m, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty(m, k, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)


def _runs_out(launch, codes):
    from tybok_b200 import ops

    lib, dev = ops._lib.load(), torch.device("cuda")
    good = launch()
    ops.check_status()
    lib.tybok_debug_set_epilogue_wait_limit(1)
    try:
        launch()
        torch.cuda.synchronize()
    finally:
        lib.tybok_debug_set_epilogue_wait_limit(0)
    assert int(ops.status_word(dev).item()) in codes
    with pytest.raises(ops._lib.TybokError, match="bounded wait"):
        ops.check_status()
    again = launch()
    ops.check_status()
    assert torch.equal(again, good)


@pytest.mark.parametrize("m,n,k,bt,splits", [(50, 1024, 4096, 0, 0), (50, 2560, 1024, 0, 0), (50, 8192, 1024, 0, 0), (300, 9600, 1024, 64, 1),
                                             (64, 128, 256, 64, 1)])
def test_one_tile_gemm(m, n, k, bt, splits):
    """K over a cluster, one full-K wave, two CTAs per SM, and a producer that is through before anyone gives up."""
    from tybok_b200 import ops

    (w8, sc), xp = _weights(n, k), ops.split3(_x(m, k), 4)
    _runs_out(lambda: ops.w8x3_linear(xp, 4, w8, sc, token_tile=bt, splits=splits)[0], (EPILOGUE,))


@pytest.mark.parametrize("m,n,k", [(1, 2560, 2048), (16, 18944, 16384)])
def test_gemm_that_makes_its_planes(m, n, k):
    from tybok_b200 import ops

    (w8, sc), x = _weights(n, k), _x(m, k)
    _runs_out(lambda: ops.w8a16_linear(x, w8, sc), (CONVERT, EPILOGUE))


@pytest.mark.parametrize("planes", [2, 3])
@pytest.mark.parametrize("m,n,k", [(300, 19072, 256), (700, 9600, 4096), (60, 38400, 1024)])
def test_pair_gemm(m, n, k, planes):
    """Several tiles per pair, K within the ring and beyond it, token tiles of two sizes, planes in columns of their own."""
    from tybok_b200 import ops

    w8, sc = _weights(n, k)
    if planes == 3:
        xp = ops.split3(_x(m, k), 4)
        _runs_out(lambda: ops.w8x3_linear(xp, 4, w8, sc)[0], (EPILOGUE,))
    else:
        xp, rs = ops.norm_planes2(_x(m, k), ops.NORM_RMS, torch.zeros(k, device="cuda"))
        _runs_out(lambda: ops.w8x2_gemm(xp, rs, w8, sc)[0], (EPILOGUE,))


def test_pair_gemm_of_two_accumulators():
    from tybok_b200 import ops

    (w8, sc), xp = _weights(16384, 1024), ops.split3(_x(500, 1024), 4)
    _runs_out(lambda: ops.w8x3_geglu_packed(xp, 4, w8, sc)[0], (EPILOGUE,))


@pytest.mark.parametrize("m,n,k", [(333, 2048, 16384), (257, 2044, 16400)])
def test_pair_gemm_that_splits_k(m, n, k):
    from tybok_b200 import ops

    (w8, sc), xp = _weights(n, k), ops.split3(_x(m, k), 4)
    _runs_out(lambda: ops.w8x3_linear(xp, 4, w8, sc)[0], (EPILOGUE,))


# one key block in a CTA; rows pushed between the CTAs of a cluster, and staged in L2; the key loop at both head sizes, with
# fewer blocks than its ring holds and more, its form of up to 64 rows, and the one of two tiles per CTA
@pytest.mark.parametrize("b,l,keys,h,g,d", [(1, 50, 100, 8, 1, 256), (1, 50, 594, 8, 1, 256), (2, 50, 594, 8, 2, 256), (1, 300, 90, 2, 1, 256),
                                            (1, 544, 544, 8, 1, 256), (1, 100, 200, 3, 3, 128), (1, 128, 1000, 24, 24, 128),
                                            (1, 50, 4146, 24, 24, 128), (1, 1000, 200, 24, 24, 128), (1, 1030, 3000, 24, 24, 128)])
def test_attention(b, l, keys, h, g, d):
    from tybok_b200 import ops

    q, k, v = _x(b * l, h * d), _x(b * g * keys, d, 1).view(b, g, keys, d), _x(b * g * keys, d, 2).view(b, g, keys, d)
    _runs_out(lambda: ops.attention(q, k, v, tokens=l, keys=keys, scale=d**-0.5)[0], (EPILOGUE,))
