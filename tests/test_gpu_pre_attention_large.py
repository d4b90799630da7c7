"""qk_norm_rope_store at sizes where the kernel works on whole tokens (full passes of eight rows), far above the line at which that
begins: bit for bit against the oracle, like the small sizes."""
import numpy as np
import pytest

from conftest import bits_to_torch, torch_to_bits
from test_gpu_pre_attention import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,h,kvh", [(3946, 32, 8), (3947, 32, 8), (5003, 32, 8), (7897, 16, 4), (7901, 12, 2), (2400, 64, 8)])
def test_large_batches_are_bit_exact(t, h, kvh):
    import torch
    from nanovllm_jax_b200 import ops
    from oracle import reference_attention as ref
    qb, kb, vb, wq, wk, cs, pos, kcb, vcb, slots = _inputs(t, h, kvh, 800 + t, nb=max(32, t // 256 + 1))
    slots[::97] = -1
    want_q, want_k = ref.qk_norm_rope(qb, kb, wq, wk, cs, pos, 1e-6)
    flat = (kcb.shape[0] * kcb.shape[1], kvh, 128)
    want_kc, want_vc = ref.store_kv_to_cache(want_k, vb, kcb.reshape(flat), vcb.reshape(flat), slots, skip_negative=True)
    q, k, v = bits_to_torch(qb), bits_to_torch(kb), bits_to_torch(vb)
    kc, vc = bits_to_torch(kcb), bits_to_torch(vcb)
    ops.qk_norm_rope_store(q, k, v, *(torch.from_numpy(x).cuda() for x in (wq, wk, cs, pos)), kc, vc,
                           torch.from_numpy(slots).cuda(), eps=1e-6)
    for got, want in ((q, want_q), (k, want_k), (v, vb), (kc, want_kc), (vc, want_vc)):
        assert np.array_equal(torch_to_bits(got).reshape(want.shape), want)
