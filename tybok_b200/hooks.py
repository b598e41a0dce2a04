"""Callables with the reference's per-module hook signatures, backed by the fp8 kernels.

The reference swaps tiers in by assigning callables onto its own model objects:
``layer.mlp.forward = fn(x[B,L,W])`` (tybok/policies/pi05/engine.py:296-298) and
``blk._fused_ffn_tail = fn(x, shift_mlp, scale_mlp, gate_mlp)``
(tybok/policies/fastwam/models/dit_block.py:205-210,392-394).  The two factories here build such
callables from a module of the reference (or anything with the same attributes), so a reference
model object can run its FFNs on this package without any other change:

    for layer in vlm.layers:
        layer.mlp.forward = make_mlp_forward(layer.mlp)
    for blk in dit.blocks:
        blk._fused_ffn_tail = make_fused_ffn_tail(blk)

Weights are read once, at construction: an ``nn.Linear``-like ``.weight`` (any float dtype, quantised
here with the reference recipe) or an ``FP8Linear``-like pair ``.weight`` (e4m3) + ``.weight_scale``.
The callables take CUDA tensors and raise for anything else; there is no CPU path.
"""

from __future__ import annotations

import torch

from . import _lib, ops
from .weights import quantize_w8


def _w8(linear, device) -> tuple[torch.Tensor, torch.Tensor]:
    w = linear.weight.detach()
    if w.dtype == torch.float8_e4m3fn:
        scale = getattr(linear, "weight_scale", None)
        if scale is None:
            raise TypeError("an e4m3 weight needs its per-output-channel `weight_scale`")
        return w.to(device).contiguous(), scale.detach().to(device).float().reshape(-1).contiguous()
    return quantize_w8(w.to(device))


def _bias(linear, device):
    b = getattr(linear, "bias", None)
    return None if b is None else b.detach().to(device, torch.bfloat16).contiguous()


def _need_cuda(x: torch.Tensor) -> None:
    if not x.is_cuda:
        raise RuntimeError("tybok_b200 hooks run on CUDA tensors only: there is no CPU path")


def make_mlp_forward(mlp, device: str | torch.device = "cuda"):
    """``fn(x [B, L, W]) -> [B, L, W]`` computing ``down(gelu_tanh(gate(x)) * up(x))`` of a
    ``GemmaMLP`` (tybok/policies/pi05/models/layers.py:87-95): bf16 -> planes, one gate/up GEMM
    whose epilogue writes the planes of the intermediate, the down projection."""
    gate, up, down = _w8(mlp.gate_proj, device), _w8(mlp.up_proj, device), _w8(mlp.down_proj, device)
    weights = (ops.pack_gate_up(*gate, *up), None, down) if gate[0].shape[0] % 64 == 0 else (gate, up, down)
    chain = _lib.native().Mlp(*weights)
    tensors = [t for w in weights for t in (w or (None, None))]

    def forward(x: torch.Tensor) -> torch.Tensor:
        _need_cuda(x)
        y = chain.forward(x) if type(x) is torch.Tensor else None  # None: the dispatcher's call
        return torch.ops.tybok_b200.mlp(x, *tensors) if y is None else y

    return forward


def make_fused_ffn_tail(blk, device: str | torch.device = "cuda"):
    """``fn(x [B, S, H], shift_mlp, scale_mlp, gate_mlp) -> [B, S, H]`` computing
    ``x + gate_mlp * ffn(modulate(norm2(x), shift_mlp, scale_mlp))`` of a ``FastWAMAttentionBlock``
    (tybok/policies/fastwam/models/dit_block.py:392-397).  The three modulation tensors hold one row
    of ``H`` values per batch element (``[B, 1, H]``, ``[1, 1, H]`` or ``[H]``; strided views of the
    ``[B, 6, H]`` table are fine); the whole batch is one launch chain."""
    up = (*_w8(blk.ffn[0], device), _bias(blk.ffn[0], device))
    down = (*_w8(blk.ffn[2], device), _bias(blk.ffn[2], device))
    eps = float(getattr(blk, "eps", 1e-6))
    chain = _lib.native().FfnTail(up, down, eps)

    def tail(x: torch.Tensor, shift_mlp: torch.Tensor, scale_mlp: torch.Tensor, gate_mlp: torch.Tensor) -> torch.Tensor:
        _need_cuda(x)
        y = chain.forward(x, shift_mlp, scale_mlp, gate_mlp) if type(x) is torch.Tensor else None
        return torch.ops.tybok_b200.ffn_tail(x, shift_mlp, scale_mlp, gate_mlp, *up, *down, eps) if y is None else y

    return tail
