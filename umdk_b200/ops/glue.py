"""Fused small kernels of the decode step (csrc/cam/decoder_glue.cu): residual add + RMSNorm, the post-processing of
the fused q_a / kv_a projection (q RMSNorm; KV RMSNorm + rotary embedding + write of the token's KV row), the rotary
part of the absorbed query, and the router (softmax + top-k + renormalisation + folded expert numbering)."""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native

# what torch.nn.functional.rms_norm uses when eps is None: the epsilon of its fp32 accumulation type
RMS_EPS = float(torch.finfo(torch.float32).eps)


def add_rmsnorm(x: torch.Tensor, w: torch.Tensor, a: Optional[torch.Tensor] = None,
                b: Optional[torch.Tensor] = None, x_out: Optional[torch.Tensor] = None,
                h: Optional[torch.Tensor] = None, eps: float = RMS_EPS) -> Tuple[torch.Tensor, torch.Tensor]:
    """(x + a + b, rmsnorm(x + a + b) * w) in one launch; with no addends the first result is ``x`` itself."""
    _native.LAUNCH_COUNT += 1
    return _native.calls().add_rmsnorm(x, w, a, b, x_out, h, eps)


def qkv_post(qkv: torch.Tensor, q_lora: int, q_norm: torch.Tensor, kv_norm: torch.Tensor, cos: torch.Tensor,
             sin: torch.Tensor, kv_pool: torch.Tensor, new_row: torch.Tensor, status: torch.Tensor,
             qa: Optional[torch.Tensor] = None, eps: float = RMS_EPS) -> torch.Tensor:
    """qkv [T, q_lora + 576] bf16 -> qa [T, q_lora]; writes row new_row[t] (int64, in rows of 576) of ``kv_pool``."""
    _native.LAUNCH_COUNT += 1
    return _native.calls().qkv_post(qkv, q_lora, q_norm, kv_norm, cos, sin, kv_pool, new_row, status, qa, eps)


def q_rope(q: torch.Tensor, nope: int, cos: torch.Tensor, sin: torch.Tensor, q_full: torch.Tensor):
    """q [T, heads, nope + 64] -> q_full[T, heads, 512:576] = rotary(q[..., nope:])."""
    _native.LAUNCH_COUNT += 1
    _native.calls().q_rope(q, nope, cos, sin, q_full)


def router_topk(logits: torch.Tensor, k: int, fold_el: int = 0, rank: int = 0):
    """logits [T, E] bf16 -> (idx [T, k(+1)] int64, w [T, k(+1)] fp32): top-k of the softmax with weights renormalised
    over the winners. ``fold_el`` > 0: ids renumbered for ranks that own fold_el routed experts plus one shared expert,
    and one more slot that selects rank ``rank``'s shared expert with weight 1 (EpLowLatency fold_shared)."""
    _native.LAUNCH_COUNT += 1
    return _native.calls().router_topk(logits, k, fold_el, rank)
