"""Prefill of few items with many keys: the K/V tiles of an item are cut into runs on several CTAs and the partial results
combined.  Around the sizes where items start to be cut (eight K/V tiles, half as many items as SMs), with prefixes that are
and are not multiples of the tile, even and odd head groups, ragged ends, a sequence too short to be cut beside one that is."""
import numpy as np
import pytest

from conftest import assert_attention_close, torch_to_bits, torch_to_f32
from test_gpu_paged_prefill import _case, _run, _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,kvh", [(4, 1), (3, 1), (1, 1), (10, 2), (16, 4)])
@pytest.mark.parametrize("prefixes,new_lens", [([5000], [100]), ([4096], [1]), ([1023, 0], [257, 3]), ([1300], [236]),
                                               ([1280], [128]), ([2047, 60, 3333], [33, 200, 1]), ([0], [1500]),
                                               ([0, 7], [1025, 900])])
def test_split_items_match_the_oracle(prefixes, new_lens, h, kvh):
    from nanovllm_jax_b200 import _lib
    c = _case(prefixes, new_lens, h=h, kvh=kvh, block_size=256, seed=900 + prefixes[0] + new_lens[0] + h, poison=True)
    a, b = _run(c), _run(c)
    assert np.array_equal(torch_to_bits(a), torch_to_bits(b))
    assert_attention_close(torch_to_f32(a), _want(c), f"{prefixes} + {new_lens} H={h} KVH={kvh}")
    assert _lib.device_status() == 0


@pytest.mark.parametrize("h,kvh,lens", [(2, 1, [3000]), (3, 1, [2100, 40]), (4, 1, [2048, 1, 1500]), (2, 2, [2050])])
def test_split_packed_prompts_match_the_oracle(h, kvh, lens):
    import torch
    from conftest import bits_to_torch
    from nanovllm_jax_b200 import _lib, ops, workloads
    from oracle import reference_attention as ref
    w = workloads.make_prefill_workload("split", seed=9500 + lens[0] + h, batch=len(lens), num_heads=h, num_kv_heads=kvh,
                                        len_lo=1, len_hi=1, seq_lens=lens)
    t = workloads.prefill_tensors_numpy(w)
    cu = torch.from_numpy(w.cu_seqlens).cuda()
    got = ops.varlen_prefill(*(bits_to_torch(t[n + "_bits"]) for n in "qkv"), cu, max(lens), w.scale,
                             cu_seqlens_host=w.cu_seqlens)
    want = ref.variable_length_attention_prefill(t["q"], t["k"], t["v"], w.cu_seqlens, w.cu_seqlens, 8192, 8192, h, kvh,
                                                 w.scale, w.batch)
    assert_attention_close(torch_to_f32(got), want, f"{lens} H={h} KVH={kvh}")
    assert _lib.device_status() == 0
