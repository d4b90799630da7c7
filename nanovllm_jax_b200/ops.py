"""Operators over torch CUDA tensors -> C ABI.  torch is used for device memory and streams only.

Every function validates dtype / device / contiguity, then hands raw device pointers to
libnvllm_b200_attn.so on torch's current stream.  Nothing here computes on the host and nothing
falls back: a missing library or an unsupported shape raises.

The checks, the buffers and the call itself are native (csrc/torch_binding.cpp); the functions below
give them their names, defaults and documentation.
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib


def workspace(device, nbytes: int) -> torch.Tensor:
    """A cached scratch buffer of at least ``nbytes`` on ``device`` (grown on demand, never shrunk).

    One buffer per (device, stream): calls on one stream are ordered, so they may share it.
    """
    index = torch.device(device).index
    return _lib.binding().workspace(torch.cuda.current_device() if index is None else index, nbytes)


def _host_lengths(x):
    """A host copy of cu_seqlens as a contiguous int32 buffer (None stays None)."""
    if x is None or (type(x) is np.ndarray and x.dtype == np.int32 and x.flags.c_contiguous):
        return x
    return torch.as_tensor(x, dtype=torch.int32, device="cpu").contiguous()


def store_kvcache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                  slot_mapping: torch.Tensor) -> None:
    """In place: ``k_cache.view(-1, KVH, D)[slot_mapping[t]] = key[t]`` (same for value).

    key/value: [T, KVH, D] bf16 or fp32.  Caches: bf16, any leading shape whose flattening is
    [num_slots, KVH, D] (e.g. [NB, block, KVH, D]).  slot_mapping: [T] int32; negative = skip.
    """
    _lib.binding().store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def paged_decode_workspace_bytes(batch: int, num_heads: int, num_kv_heads: int, head_dim: int, max_blocks: int,
                                 block_size: int, device=None) -> int:
    with torch.cuda.device(device):
        return int(_lib.load().nvllm_b200_paged_decode_workspace_bytes(batch, num_heads, num_kv_heads, head_dim,
                                                                       max_blocks, block_size))


def paged_decode(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, block_tables: torch.Tensor,
                 context_lens: torch.Tensor, scale: float, block_size: int, out: torch.Tensor | None = None,
                 scratch: torch.Tensor | None = None) -> torch.Tensor:
    """Decode attention over the paged cache; returns [B, H, D] bf16."""
    return _lib.binding().paged_decode(q, k_cache, v_cache, block_tables, context_lens, scale, block_size, out, scratch)


def decode_step(q: torch.Tensor, key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                slot_mapping: torch.Tensor, block_tables: torch.Tensor, context_lens: torch.Tensor, scale: float,
                block_size: int, out: torch.Tensor | None = None) -> torch.Tensor:
    """One decode step of one layer in one C call: scatter key/value [B, KVH, D] into the cache by slot, then
    attend (same result as ``store_kvcache`` followed by ``paged_decode``).  Caches are [NB, block, KVH, D]."""
    return _lib.binding().decode_step(q, key, value, k_cache, v_cache, slot_mapping, block_tables, context_lens, scale,
                                      block_size, out, False)


def varlen_prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens: torch.Tensor, max_seqlen: int,
                   scale: float, out: torch.Tensor | None = None, cu_seqlens_host=None,
                   cu_seqlens_k: torch.Tensor | None = None) -> torch.Tensor:
    """Causal attention over packed sequences; returns [T, H, D] bf16.

    ``cu_seqlens_host`` (a CPU int32 tensor / numpy array equal to ``cu_seqlens``) lets the library size its
    grid exactly without a device read; without it the grid is sized from ``max_seqlen``.
    """
    return _lib.binding().varlen_prefill(q, k, v, cu_seqlens, max_seqlen, scale, out, _host_lengths(cu_seqlens_host),
                                         cu_seqlens_k)


def paged_prefill(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, block_tables: torch.Tensor,
                  cu_seqlens_q: torch.Tensor, cu_seqlens_k: torch.Tensor, max_seqlen_q: int, scale: float,
                  block_size: int, out: torch.Tensor | None = None, cu_seqlens_host=None) -> torch.Tensor:
    """Causal attention of packed new tokens over their whole sequences (cached prefix included), keys/values read from
    the paged cache [NB, block, KVH, D] through ``block_tables``; returns [T, H, D] bf16.  The new tokens' K/V rows
    must already be in the cache."""
    return _lib.binding().paged_prefill(q, k_cache, v_cache, block_tables, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, scale,
                                        block_size, out, _host_lengths(cu_seqlens_host))


def qk_norm_rope_store(q: torch.Tensor, key: torch.Tensor, value: torch.Tensor, q_weight: torch.Tensor,
                       k_weight: torch.Tensor, cos_sin_cache: torch.Tensor, positions: torch.Tensor,
                       k_cache: torch.Tensor, v_cache: torch.Tensor, slot_mapping: torch.Tensor, eps: float = 1e-6) -> None:
    """In place, one pass: per-head RMSNorm of q and key, rotary embedding of both, scatter of the rotated key rows and
    the value rows into the cache by slot.  Caches: any leading shape whose flattening is [num_slots, KVH, D]."""
    _lib.binding().qk_norm_rope_store(q, key, value, q_weight, k_weight, cos_sin_cache, positions, k_cache, v_cache,
                                      slot_mapping, eps)


def fused_decode_step(q: torch.Tensor, key: torch.Tensor, value: torch.Tensor, q_weight: torch.Tensor,
                      k_weight: torch.Tensor, cos_sin_cache: torch.Tensor, positions: torch.Tensor,
                      k_cache: torch.Tensor, v_cache: torch.Tensor, slot_mapping: torch.Tensor,
                      block_tables: torch.Tensor, context_lens: torch.Tensor, scale: float, block_size: int,
                      eps: float = 1e-6, out: torch.Tensor | None = None) -> torch.Tensor:
    """``qk_norm_rope_store`` (q and key updated in place) followed by ``paged_decode``, as one C call and two kernel
    launches; returns the attention output [B, H, D]."""
    return _lib.binding().fused_decode_step(q, key, value, q_weight, k_weight, cos_sin_cache, positions, k_cache, v_cache,
                                            slot_mapping, block_tables, context_lens, scale, block_size, eps, out)
