"""Long lists whose keys and values do not fit the L2: the kv heads are taken in groups.  Every sequence must come out as it does
alone (one group), bit for bit; lengths just below and above the size at which a second group begins (96 MiB of K and V: 196 608
(token, kv head) rows) and a fourth (twice that, and six rounds of items per SM and group)."""
import numpy as np
import pytest

from conftest import torch_to_bits

pytestmark = pytest.mark.gpu


def _groups(lens, h, kvh, sms):
    span, n = 128 // (h // kvh // 2), 1  # tokens of an item (even numbers of q heads per kv head)
    items = sum(-(-x // span) for x in lens) * kvh
    while kvh % (2 * n) == 0 and sum(lens) * kvh > 196608 * n and items >= 2 * n * 6 * sms:
        n *= 2
    return n


@pytest.mark.parametrize("h,kvh,tokens,groups", [(32, 8, 24575, 1), (32, 8, 24577, 2), (48, 12, 33000, 4), (16, 8, 54500, 2),
                                                 (16, 8, 55000, 4), (40, 5, 40000, 1)])
def test_sequences_come_out_as_they_do_alone(h, kvh, tokens, groups):
    import torch
    from nanovllm_jax_b200 import _lib, ops
    lens = [1, 4000, 129, 2500, 777, 3000]
    while sum(lens) < tokens:
        lens.append(min(1500 + 37 * len(lens), tokens - sum(lens)))
    assert _groups(lens, h, kvh, torch.cuda.get_device_properties(0).multi_processor_count) == groups
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn((tokens, n, 128), generator=gen, device="cuda", dtype=torch.bfloat16) for n in (h, kvh, kvh))
    got = ops.varlen_prefill(q, k, v, torch.from_numpy(cu).cuda(), max(lens), 128 ** -0.5, cu_seqlens_host=cu)
    for b in (0, 1, 2, len(lens) // 2, len(lens) - 1):
        a, z = cu[b], cu[b + 1]
        one = np.asarray([0, z - a], np.int32)
        want = ops.varlen_prefill(q[a:z], k[a:z], v[a:z], torch.from_numpy(one).cuda(), int(z - a), 128 ** -0.5,
                                  cu_seqlens_host=one, out=torch.empty_like(q[a:z]))
        assert np.array_equal(torch_to_bits(got[a:z]), torch_to_bits(want)), f"sequence {b}"
    assert _lib.device_status() == 0
