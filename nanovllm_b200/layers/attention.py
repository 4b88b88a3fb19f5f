"""Drop-in replacement for nano-vllm's attention layer (nanovllm/layers/attention.py).

Same surface as the reference: `store_kvcache(key, value, k_cache, v_cache, slot_mapping)` and
`Attention(num_heads, head_dim, scale, num_kv_heads).forward(q, k, v)`, the per-step metadata
read from `get_context()` (nanovllm/utils/context.py), the cache bound by the model runner onto
`k_cache` / `v_cache` with layout (num_blocks, block_size, num_kv_heads, head_dim)
(nanovllm/engine/model_runner.py:107-117).  The arithmetic runs in hand-written sm_100a CUDA
behind the C ABI of include/b200_attn.h; tensor checks, output allocation and the call into it are compiled too
(csrc/native.cpp): done in Python they took longer than the kernels of a small step.  There is no Triton, no
flash_attn and no fallback.
"""
from __future__ import annotations

import torch
from torch import nn

from .. import _lib
from ..utils import context as _own_context

# The function the layer reads its metadata from.  nanovllm_b200.integration rebinds it to the
# reference engine's get_context when the layer is installed into nano-vllm.
_context_getter = _own_context.get_context

def get_context():
    return _context_getter()


def set_context_getter(fn):
    global _context_getter
    _context_getter = fn


def store_kvcache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                  slot_mapping: torch.Tensor):
    """Same contract and asserts as the reference wrapper (nanovllm/layers/attention.py:33-40)."""
    _lib.native().store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def decode_attention(q, k_cache, v_cache, context_lens, block_tables, scale, num_kv_heads):
    """q (B, H, D) -> (B, 1, H, D), the shape flash_attn_with_kvcache returns for the reference's
    call (nanovllm/layers/attention.py:72-74).  The kernel's workspace is one zero-initialised tensor per
    (device, query heads per kv head), allocated on first use (the engine's eager warm-up precedes graph capture)."""
    return _lib.native().decode_attention(q, k_cache, v_cache, context_lens, block_tables, scale, num_kv_heads)


def prefill_attention(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale, num_kv_heads,
                      block_tables=None, kernel_variant=0):
    """Varlen causal attention.  With block_tables, k and v are the paged caches
    (nanovllm/layers/attention.py:65-70); otherwise packed (total_k, Hkv, D) activations."""
    return _lib.native().prefill_attention(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale,
                                           num_kv_heads, block_tables, kernel_variant)


class Attention(nn.Module):
    """Constructor, attributes and forward of the reference module
    (nanovllm/layers/attention.py:43-75); the model runner finds the layer through its
    `k_cache` / `v_cache` attributes (nanovllm/engine/model_runner.py:113-117)."""

    def __init__(self, num_heads, head_dim, scale, num_kv_heads):
        super().__init__()
        self.num_heads = num_heads
        self.head_dim = head_dim
        self.scale = scale
        self.num_kv_heads = num_kv_heads
        self.k_cache = self.v_cache = torch.tensor([])

    def forward(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, already_stored: bool = False):
        """`already_stored` is not part of the reference's signature: the fused producer kernel
        (layers/qk_norm_rope.py) has written k and v to the cache and passes True."""
        return _lib.native().attention_forward(q, k, v, self.k_cache, self.v_cache, _context_getter(), self.scale,
                                               self.num_kv_heads, already_stored)
