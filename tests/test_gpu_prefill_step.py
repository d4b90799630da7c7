"""Attention.__call__ on a prefill step as one C call (nvllm_b200_prefill_step): wherever the K/V scatter runs -- CTAs of
its own beside a short list of items, or a launch in front, with the plan kernel working beside it -- the
caches equal the oracle's bit for bit and the output equals the attention entry points' and, at small sizes, the oracle's.
The group sizes include odd ones (a Q tile holds all heads and half of an item's tokens; in the others half of the heads)."""
import math

import numpy as np
import pytest

from conftest import assert_attention_close, bits_to_torch, torch_to_bits, torch_to_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,kvh", [(8, 2), (10, 2), (3, 1), (7, 1), (4, 4), (32, 8)])
@pytest.mark.parametrize("lens,host", [([1], True), ([87], True), ([87], False), ([128, 129], True), ([300, 5, 256, 257, 31], True),
                                       ([300, 5, 256, 257, 31], False), ([290] * 10, True), ([20] * 200, True),
                                       ([385, 640, 17] * 14, True), ([3000] * 4 + [77], True)])
def test_store_and_attend_in_one_call(lens, host, h, kvh):
    import torch
    from nanovllm_jax_b200 import _lib, ops, workloads
    from nanovllm_jax_b200.layers.attention import Attention
    from nanovllm_jax_b200.utils.context import create_prefill_context
    from oracle import reference_attention as ref
    w = workloads.make_prefill_workload("step", seed=8000 + len(lens) + lens[0] + h, batch=len(lens), num_heads=h,
                                        num_kv_heads=kvh, len_lo=1, len_hi=1, seq_lens=lens)
    t = workloads.prefill_tensors_numpy(w)
    w.slot_mapping[::41] = -1
    shape = (w.num_blocks, w.block_size, kvh, 128)
    flat = (w.num_blocks * w.block_size, kvh, 128)
    before = np.full(flat, 0x3F80, np.uint16)
    want_k, want_v = ref.store_kv_to_cache(t["k_bits"], t["v_bits"], before, before, w.slot_mapping, skip_negative=True)
    attn = Attention(h, 128, w.scale, kvh, w.block_size)
    attn.set_kv_cache(bits_to_torch(before).view(shape), bits_to_torch(before).view(shape))
    q, k, v = (bits_to_torch(t[n + "_bits"]) for n in "qkv")
    cu = torch.from_numpy(w.cu_seqlens).cuda()
    ctx = create_prefill_context(cu, cu, max(lens), max(lens), torch.from_numpy(w.slot_mapping).cuda(),
                                 cu_seqlens_host=w.cu_seqlens if host else None)
    got = attn(q, k, v, ctx)
    assert np.array_equal(torch_to_bits(attn.k_cache).reshape(flat), want_k)
    assert np.array_equal(torch_to_bits(attn.v_cache).reshape(flat), want_v)
    alone = ops.varlen_prefill(q, k, v, cu, ctx.max_seqlen_q, w.scale)
    assert np.array_equal(torch_to_bits(got), torch_to_bits(alone))
    if w.total_tokens <= 1200:
        want = ref.variable_length_attention_prefill(t["q"], t["k"], t["v"], w.cu_seqlens, w.cu_seqlens, 8192, 8192, h, kvh,
                                                     w.scale, w.batch)
        assert_attention_close(torch_to_f32(got), want, f"{lens} H={h} KVH={kvh}")
    assert _lib.device_status() == 0


def test_long_sequences_store_and_attend_again_and_again():
    """Eight sequences of 3000 tokens, several calls in a row: the plan of a call runs beside its scatter, and the scatter
    may start while the call in front of it still attends."""
    test_store_and_attend_in_one_call([3000] * 8, True, 16, 2)
    test_store_and_attend_in_one_call([3000] * 8, False, 16, 2)
