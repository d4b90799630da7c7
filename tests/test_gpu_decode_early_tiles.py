"""The decode kernel requests its first tiles before the kernel that stores the step's K/V rows has finished, except tiles
that hold a slot of the step.  Here the step's slots lie anywhere -- in the first tile of other sequences too -- and the
one-call step must still equal the store followed by the attention, bit for bit, and the oracle."""
import math

import numpy as np
import pytest

from conftest import assert_attention_close, bits_to_torch, torch_to_bits, torch_to_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,ctx_hi", [(1, 40), (1, 3000), (5, 700), (33, 260), (256, 90), (257, 90), (600, 70)])
@pytest.mark.parametrize("h,kvh", [(8, 1), (10, 2)])
def test_step_slots_in_tiles_requested_early(batch, ctx_hi, h, kvh):
    import torch
    from nanovllm_jax_b200 import _lib, ops, workloads
    from oracle import reference_attention as ref
    block = 64 if batch > 33 else 128
    rng = np.random.Generator(np.random.PCG64(7000 + batch + ctx_hi + h))
    ctx = rng.integers(1, ctx_hi + 1, batch).astype(np.int32)
    ctx[rng.integers(0, batch)] = ctx_hi
    need = -(-ctx // block)
    nb = int(need.sum()) + 2
    perm = rng.permutation(nb).astype(np.int32)
    tables = np.full((batch, int(need.max())), -1, np.int32)
    live = []
    for b, at in enumerate(np.concatenate([[0], np.cumsum(need)[:-1]])):
        tables[b, :need[b]] = perm[at:at + need[b]]
        live.append(tables[b, 0] * block + rng.integers(0, min(block, ctx[b])))  # a row of the first page
    slots = np.asarray(live, np.int32)[rng.permutation(batch)]  # ... of some sequence, not of its own
    slots[rng.integers(0, batch)] = -1 if batch > 1 else slots[0]
    q, qb = workloads.normal_bf16_numpy(rng, (batch, h, 128))
    k_new, knb = workloads.normal_bf16_numpy(rng, (batch, kvh, 128))
    v_new, vnb = workloads.normal_bf16_numpy(rng, (batch, kvh, 128))
    _, kcb = workloads.normal_bf16_numpy(rng, (nb, block, kvh, 128))
    _, vcb = workloads.normal_bf16_numpy(rng, (nb, block, kvh, 128))
    flat = (nb * block, kvh, 128)
    want_k, want_v = ref.store_kv_to_cache(k_new, v_new, kcb.reshape(flat), vcb.reshape(flat), slots, skip_negative=True)
    scale = 1 / math.sqrt(128)
    want = ref.paged_decode_attention_streamed(q, want_k.reshape(kcb.shape), want_v.reshape(vcb.shape), tables, ctx, scale,
                                               block, kv_dtype_bits=True)
    dev = [torch.from_numpy(x).cuda() for x in (slots, tables, ctx)]
    two_k, two_v = bits_to_torch(kcb), bits_to_torch(vcb)
    ops.store_kvcache(bits_to_torch(knb), bits_to_torch(vnb), two_k, two_v, dev[0])
    two = ops.paged_decode(bits_to_torch(qb), two_k, two_v, dev[1], dev[2], scale, block)
    for _ in range(3):  # back to back, as a serving loop calls it
        kc, vc = bits_to_torch(kcb), bits_to_torch(vcb)
        one = ops.decode_step(bits_to_torch(qb), bits_to_torch(knb), bits_to_torch(vnb), kc, vc, dev[0], dev[1], dev[2],
                              scale, block)
        assert np.array_equal(torch_to_bits(kc).reshape(flat), want_k) and np.array_equal(torch_to_bits(vc).reshape(flat), want_v)
        assert np.array_equal(torch_to_bits(one), torch_to_bits(two))
    assert_attention_close(torch_to_f32(one), want, f"batch {batch}")
    assert _lib.device_status() == 0
