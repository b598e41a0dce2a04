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
