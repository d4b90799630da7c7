"""Short questions behind long cached conversations: the items that are cut into runs are of one Q tile where that leaves the runs
about as short as items of two would, and of two elsewhere.  At lengths around a tile's tokens and an item's, behind prefixes on
both sides of the rule; block tables that are padded far beyond the longest sequence take the call to the other side."""
import numpy as np
import pytest

from conftest import assert_attention_close, torch_to_bits, torch_to_f32
from test_gpu_paged_prefill import _case, _run, _want
from test_gpu_prefill_packed_heads import _pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,kvh", [(1, 1), (2, 1), (3, 1), (4, 2), (5, 1), (7, 1), (8, 1), (11, 1), (16, 1), (4, 8), (2, 8)])
@pytest.mark.parametrize("prefixes,behind", [([1100], 0), ([2600], 1), ([6400], 0), ([895, 1500], -1)])
@pytest.mark.parametrize("padded", [False, True])
def test_questions_behind_prefixes_match_the_oracle(group, kvh, prefixes, behind, padded):
    from nanovllm_jax_b200 import _lib
    tokens, span = _pack(group)
    new = [min(span, 1000) + behind, max(1, tokens + behind - 20)][:len(prefixes)]
    c = _case(prefixes, new, h=group * kvh, kvh=kvh, block_size=256, seed=6200 + group + kvh + prefixes[0], poison=True)
    if padded:
        c["tables"] = np.pad(c["tables"], ((0, 0), (0, 200)), constant_values=-1)
    a, b = _run(c), _run(c)
    assert np.array_equal(torch_to_bits(a), torch_to_bits(b))
    assert_attention_close(torch_to_f32(a), _want(c), f"{group} x {kvh}: {prefixes} + {new}")
    assert _lib.device_status() == 0
