"""Producer side of the attention layer as one CUDA launch: per-head RMSNorm of q and k, rotary
embedding, and the cache store -- the work nano-vllm does between its fused qkv projection and its
attention call (nanovllm/models/qwen3.py:75-79 plus the store at nanovllm/layers/attention.py:62-63).

`qk_norm_rope_store` is the operator; `fused_attention_forward` is a drop-in body for
`Qwen3Attention.forward` (nanovllm/models/qwen3.py:68-82) that uses it and then calls this package's
attention with the store already done.  Everything runs through libb200attn's C ABI; there is no
fallback.
"""
from __future__ import annotations

import torch

from .. import _lib
from . import attention as _attn


def qk_norm_rope_store(qkv: torch.Tensor, positions: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor,
                       cos_sin_cache: torch.Tensor, eps: float, num_heads: int, num_kv_heads: int,
                       k_cache: torch.Tensor | None = None, v_cache: torch.Tensor | None = None,
                       slot_mapping: torch.Tensor | None = None):
    """qkv (N, (H + 2 Hkv) * 128) bf16 -> (q (N, H, 128), k (N, Hkv, 128), v view (N, Hkv, 128)).
    q and k are normalised and rotated exactly in the reference's order of operations; with caches
    given, k and v of token i are also written to flat cache row slot_mapping[i] (-1: skipped)."""
    return _lib.native().qk_norm_rope_store(qkv, positions, q_weight, k_weight, cos_sin_cache, eps, num_heads, num_kv_heads,
                                            k_cache, v_cache, slot_mapping)


def fused_attention_forward(self, positions: torch.Tensor, hidden_states: torch.Tensor) -> torch.Tensor:
    """Body for `Qwen3Attention.forward` (nanovllm/models/qwen3.py:68-82): same inputs, same output,
    with q_norm, k_norm, rotary_emb and the cache store done by one kernel."""
    qkv = self.qkv_proj(hidden_states)
    attn = self.attn
    context = _attn.get_context()
    q, k, v = qk_norm_rope_store(qkv, positions, self.q_norm.weight, self.k_norm.weight,
                                 self.rotary_emb.cos_sin_cache, self.q_norm.eps, self.num_heads, self.num_kv_heads,
                                 attn.k_cache, attn.v_cache, context.slot_mapping)
    o = attn.forward(q, k, v, already_stored=True)
    return self.o_proj(o.flatten(1, -1))
