"""What the native chains refuse before they launch anything.  The checks come before the test for a CUDA tensor, so they
run here: a call whose sizes agree ends in ``NotImplementedError`` (there is no CPU path), any other in its own error."""

import pytest
import torch

HEADS, HD, H, FFN, M, LV, C = 2, 128, 256, 512, 9, 130, 21
A = HEADS * HD


def _bf(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


def _w(n, k, bias=True):
    return (torch.zeros(n, k, dtype=torch.uint8), torch.ones(n), *([_bf(n)] if bias else []))


def _dit_block():
    from tybok_b200 import _lib

    return _lib.native().DitBlock(HEADS, HD, 1e-6, _w(3 * A, H), _w(H, A), _w(A, H), _w(H, A), _w(FFN, H), _w(H, FFN), _bf(A),
                                  _bf(A), _bf(A), _bf(H), _bf(H))


def _block_args(**over):
    args = dict(x=_bf(M, H), mods=_bf(6, H), cos=torch.zeros(M, HD // 2), sin=torch.zeros(M, HD // 2), k_cache=_bf(HEADS, 256, HD),
                v_cache=_bf(HEADS, 256, HD), key_off=0, k_rows=_bf(LV, A), v_rows=_bf(LV, A), cross_k=_bf(C, A), cross_v=_bf(C, A),
                valid=torch.ones(1, C, dtype=torch.uint8))
    args.update(over)
    return list(args.values())


@pytest.mark.parametrize("over", [
    dict(),
    dict(cross_k=_bf(C + 3, A), cross_v=_bf(C + 3, A)),  # keys past the end of the mask are not read
    dict(cross_k=_bf(1, HEADS, C, HD), cross_v=_bf(1, HEADS, C, HD)),
    dict(k_rows=None, v_rows=None, k_cache=_bf(1, HEADS, M, HD), v_cache=_bf(1, HEADS, M, HD)),
    dict(cross_k=None, cross_v=None, valid=None),
    dict(mods=_bf(6, 2 * H)[:, :H]),  # rows of a wider table
])
def test_dit_block_takes_agreeing_sizes(over):
    with pytest.raises(NotImplementedError, match="no CPU implementation"):
        _dit_block().forward(*_block_args(**over))


@pytest.mark.parametrize("over", [
    dict(cross_k=_bf(C - 1, A), cross_v=_bf(C - 1, A)),  # the mask's length is the number of rows the kernel reads
    dict(cross_k=_bf(1, HEADS, C - 1, HD), cross_v=_bf(1, HEADS, C - 1, HD)),
    dict(cross_v=_bf(C - 1, A)),
    dict(cross_v=None),
    dict(cross_v=_bf(1, HEADS, C, HD)),
    dict(v_rows=_bf(LV - 1, A)),
    dict(v_rows=None),
    dict(k_rows=None),
    dict(v_cache=_bf(HEADS, 255, HD)),
    dict(k_cache=_bf(2, HEADS, 256, HD)),
    dict(valid=torch.ones(2, C, dtype=torch.uint8)),
])
def test_dit_block_refuses_disagreeing_sizes(over):
    with pytest.raises((TypeError, ValueError)):
        _dit_block().forward(*_block_args(**over))


def test_token_rows_of_another_count_are_refused():
    from tybok_b200.dit import _token_rows

    assert _token_rows(_bf(1, LV, A), LV, A).shape == (LV, A)
    assert _token_rows(torch.zeros(LV, A + 1)[:, 1:], LV, A).is_contiguous()
    for bad in (_bf(2, LV, A), _bf(1, LV, 2 * A), _bf(1, LV - 1, A)):
        with pytest.raises(ValueError):
            _token_rows(bad, LV, A)


def _meta(t):
    """The tensor on another device than the rest of the call."""
    return t.to("meta")


def _gemma(w=256, inner=512, heads=2, g=1, hd=128, norms=True, layers=2):
    from tybok_b200 import _lib

    n = (torch.zeros(w), torch.zeros(w)) if norms else (None, None)
    lay = lambda: (_w((heads + 2 * g) * hd, w, False), _w(w, heads * hd, False), _w(2 * inner, w, False), None,  # noqa: E731
                   _w(w, inner, False), *n)
    return _lib.native().GemmaStack(w, heads, g, hd, [lay() for _ in range(layers)])


def _gemma_args(b=1, l=7, w=256, g=1, hd=128, layers=2, **over):
    args = dict(x=_bf(b * l, w), b=b, l=l, pos=torch.zeros(b * l, dtype=torch.int32), cos=_bf(40, hd), sin=_bf(40, hd),
                kc=[_bf(b, g, 20, hd) for _ in range(layers)], vc=[_bf(b, g, 20, hd) for _ in range(layers)], key_off=3,
                key_valid=torch.ones(b, 3 + l, dtype=torch.uint8), mods=None, fold=None, first=0, count=layers, wait=[], record=[])
    args.update(over)
    return list(args.values())


@pytest.mark.parametrize("name", ["x", "mods", "cos", "k_cache", "v_cache", "k_rows", "v_rows", "cross_k", "cross_v", "valid"])
def test_dit_block_refuses_a_tensor_of_another_device(name):
    good = dict(zip(("x", "mods", "cos", "sin", "k_cache", "v_cache", "key_off", "k_rows", "v_rows", "cross_k", "cross_v", "valid"),
                    _block_args()))
    with pytest.raises(ValueError, match="tensors on"):
        _dit_block().forward(*_block_args(**{name: _meta(good[name])}))


@pytest.mark.parametrize("over", [dict(pos=_meta(torch.zeros(7, dtype=torch.int32))), dict(key_valid=_meta(torch.ones(1, 10, dtype=torch.uint8))),
                                  dict(kc=[_bf(1, 1, 20, 128), _meta(_bf(1, 1, 20, 128))]), dict(x=_meta(_bf(7, 256)))])
def test_gemma_stack_refuses_a_tensor_of_another_device(over):
    with pytest.raises(NotImplementedError):
        _gemma().forward(*_gemma_args())
    with pytest.raises(ValueError, match="tensors on"):
        _gemma().forward(*_gemma_args(**over))


def test_calls_and_weights_of_another_device_are_refused():
    from tybok_b200 import _lib, ops

    nat = _lib.native()
    up, down = _w(FFN, H), _w(H, FFN)
    mod = _bf(1, H)
    calls = [
        lambda: ops.w8a16_linear(_bf(3, H), *up[:2], _meta(up[2])),
        lambda: ops.w8a16_linear(_bf(3, H), _meta(up[0]), up[1]),
        lambda: ops.attention(_bf(4, 128), _bf(1, 1, 9, 128), _meta(_bf(1, 1, 9, 128)), tokens=4, keys=9, scale=1.0),
        lambda: nat.Mlp(up, None, _w(H, FFN // 2)).forward(_meta(_bf(3, H))),
        lambda: nat.FfnTail(up, down, 1e-6).forward(_bf(3, H), mod, mod, _meta(mod)),
        lambda: nat.FfnTail(up, tuple(map(_meta, down)), 1e-6),
        lambda: nat.FfnTail((up[0], _meta(up[1])), down, 1e-6),
    ]
    for call in calls:
        with pytest.raises(ValueError, match="tensors on"):
            call()


@pytest.mark.parametrize("over", [
    dict(cos=torch.zeros(HD // 2, M)), dict(mods=_bf(5, H)), dict(x=_bf(M, H + 16)),
])
def test_dit_block_refuses_other_shapes(over):
    with pytest.raises((TypeError, ValueError)):
        _dit_block().forward(*_block_args(**over))


@pytest.mark.parametrize("i,bad", [(3, _w(3 * A, H + 16)), (4, _w(H, A + 128)), (5, _w(A + 128, H)), (6, _w(H + 128, A)), (7, _w(FFN, H + 16)),
                                   (8, _w(H, FFN + 16)), (9, _bf(A - 8)), (12, _bf(H + 8)), (13, torch.zeros(H))])
def test_dit_block_refuses_weights_that_disagree(i, bad):
    from tybok_b200 import _lib

    args = [HEADS, HD, 1e-6, _w(3 * A, H), _w(H, A), _w(A, H), _w(H, A), _w(FFN, H), _w(H, FFN), _bf(A), _bf(A), _bf(A), _bf(H), _bf(H)]
    _lib.native().DitBlock(*args)
    args[i] = bad
    with pytest.raises((TypeError, ValueError)):
        _lib.native().DitBlock(*args)


@pytest.mark.parametrize("i,bad", [(0, _w(512, 272, False)), (0, _w(640, 256, False)), (1, _w(256, 384, False)), (2, _w(1024, 272, False)),
                                   (2, _w(1152, 256, False)), (4, _w(384, 512, False)), (4, _w(256, 640, False)), (5, torch.zeros(264))])
def test_gemma_stack_refuses_weights_that_disagree(i, bad):
    from tybok_b200 import _lib

    lay = [_w(512, 256, False), _w(256, 256, False), _w(1024, 256, False), None, _w(256, 512, False), torch.zeros(256), torch.zeros(256)]
    other = list(lay)
    other[i] = bad
    _lib.native().GemmaStack(256, 2, 1, 128, [tuple(lay), tuple(lay)])
    with pytest.raises((TypeError, ValueError)):
        _lib.native().GemmaStack(256, 2, 1, 128, [tuple(lay), tuple(other)])


def test_gemma_stack_refuses_calls_that_disagree():
    mod = lambda n=768: [(torch.zeros(1, n), torch.zeros(1, n))] * 2  # noqa: E731
    fold = lambda q=512, gu=1024: [(torch.zeros(q), torch.zeros(gu))] * 2  # noqa: E731
    with pytest.raises(NotImplementedError):
        _gemma(norms=False).forward(*_gemma_args(mods=mod(), fold=fold()))
    for over in (dict(fold=fold(q=504)), dict(fold=fold(gu=512)), dict(mods=mod(512)), dict(mods=None), dict(wait=[0]), dict(record=[0]),
                 dict(sin=_bf(39, 128)), dict(kc=[_bf(1, 1, 20, 128), _bf(1, 1, 19, 128)]), dict(kc=[_bf(20, 128)] * 2)):
        with pytest.raises((TypeError, ValueError)):
            _gemma(norms=False).forward(*_gemma_args(**{**dict(mods=mod(), fold=fold()), **over}))


def test_single_calls_refuse_disagreeing_operands():
    from tybok_b200 import _lib, ops

    nat = _lib.native()
    w, s, b = _w(FFN, H)
    kv = _bf(1, 1, 9, 128)
    for good in (lambda: ops.w8a16_linear(_bf(3, H), w, s, b, epilogue=ops.EPI_RESIDUAL, residual=_bf(3, FFN), gate=_bf(2, FFN), rows_per_gate=2),
                 lambda: ops.attention(_bf(4, 256), kv, kv, tokens=4, keys=9, scale=1.0)):
        with pytest.raises(NotImplementedError):
            good()
    calls = [
        lambda: ops.w8a16_linear(_bf(3, H), w, s, b.float()),
        lambda: ops.w8a16_linear(_bf(3, H), w, s, _bf(FFN - 4)),
        lambda: ops.w8a16_linear(_bf(3, H), w, s, epilogue=ops.EPI_RESIDUAL, residual=_bf(3, FFN), gate=_bf(1, FFN), rows_per_gate=2),
        lambda: ops.attention(_bf(4, 256), kv, _bf(1, 1, 8, 128), tokens=4, keys=9, scale=1.0),
        lambda: ops.attention(_bf(4, 256), kv, kv.float(), tokens=4, keys=9, scale=1.0),
        lambda: ops.attention(_bf(4, 256), kv.transpose(2, 3).contiguous().transpose(2, 3), kv, tokens=4, keys=9, scale=1.0),
        lambda: ops.attention(_bf(4, 192), kv, kv, tokens=4, keys=9, scale=1.0),
        lambda: nat.Mlp(_w(FFN, H, False), _w(FFN, H + 16, False), _w(H, FFN, False)),
        lambda: nat.FfnTail(_w(FFN, H), _w(H, FFN + 16), 1e-6),
    ]
    for call in calls:
        with pytest.raises((TypeError, ValueError)):
            call()


def test_attention_workspace_of_the_form_that_is_taken():
    """Many clusters over one key head, several query tiles and head_dim 128 exchange nothing; what is needed is never more
    than the bound that knows neither heads nor head size."""
    from tybok_b200 import _lib

    lib = _lib.load()
    need = lib.tybok_attention_workspace_needed
    one = need(1, 50, 8, 1, 256, 594)
    assert one == lib.tybok_attention_workspace_bytes(1, 50, 8, 594) == 2 * 5 * 8 * (128 * 256 * 4 + 128 * 8)
    assert need(32, 50, 8, 1, 256, 594) == 0 < lib.tybok_attention_workspace_bytes(32, 50, 8, 594)
    assert need(32, 50, 8, 2, 256, 594) == 32 * one
    assert need(1, 50, 8, 1, 256, 128) == need(1, 129, 8, 8, 256, 594) == need(1, 50, 24, 24, 128, 4146) == 0
    for b in range(1, 40):
        for keys in (100, 129, 594, 1024):
            assert need(b, 50, 8, 1, 256, keys) <= lib.tybok_attention_workspace_bytes(b, 50, 8, keys)
