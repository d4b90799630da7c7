"""A sequence's result depends on its own tokens alone.  Q tiles hold the next sequence's first queries behind a sequence's end; here
their scores grow by far more than the rescale threshold from one K/V tile to the next, beside rows whose scores hardly move, and
the sequence must come out as it does alone, bit for bit."""
import numpy as np
import pytest

from conftest import torch_to_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 2, 4, 5, 7, 8])
@pytest.mark.parametrize("length", [261, 777, 900])
def test_scores_of_the_sequence_behind_do_not_matter(group, length):
    import torch
    from nanovllm_jax_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(6100 + length + group)
    lens = [length, 300]
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    q, k, v = (torch.randn((sum(lens), n, 128), generator=gen, device="cuda", dtype=torch.bfloat16) for n in (group, 1, 1))
    q[length:] *= 200

    def run(n, count):
        return ops.varlen_prefill(q[:n], k[:n], v[:n], torch.from_numpy(cu[:count + 1]).cuda(), max(lens[:count]), 128 ** -0.5,
                                  cu_seqlens_host=cu[:count + 1], out=torch.empty_like(q[:n]))

    assert np.array_equal(torch_to_bits(run(length, 1)), torch_to_bits(run(sum(lens), 2)[:length]))
    assert _lib.device_status() == 0
