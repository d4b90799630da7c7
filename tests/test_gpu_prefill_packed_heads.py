"""Q tiles of (token, head) rows: every number of q heads per kv head, at lengths around the tokens of a tile and of an item,
with prefixes that put the last key at and around the steps of 16 keys that a tile's products go through, garbage behind the
sequences' ends, and runs of two K/V tiles."""
import numpy as np
import pytest

from conftest import assert_attention_close, torch_to_bits, torch_to_f32
from test_gpu_paged_prefill import _case, _run, _want

pytestmark = pytest.mark.gpu


def _pack(group):
    w = max(x for x in range(1, 9) if group % x == 0)
    tokens = 128 // (w if w % 2 else w // 2)
    return tokens, 2 * tokens if w % 2 else tokens


@pytest.mark.parametrize("group,kvh", [(1, 2), (2, 1), (3, 2), (4, 1), (5, 1), (6, 2), (7, 1), (8, 1), (9, 1), (10, 1), (11, 1),
                                       (16, 1)])
@pytest.mark.parametrize("around", ["tile", "item", "steps"])
def test_packed_rows_match_the_oracle(group, kvh, around):
    from nanovllm_jax_b200 import _lib
    tokens, span = _pack(group)
    if around == "steps":
        prefixes, new = [0, 1, 14, 15, 16, 17, 112, 127, 128, 1090], [16, 16, 1, 1, 1, 31, 16, 1, 17, 3]
    else:
        at = tokens if around == "tile" else span
        new, prefixes = [at - 1, at, at + 1, 2 * at, 2 * at + 1], [0, 0, 127, 128 - at % 128, 900]
    c = _case(prefixes, new, h=group * kvh, kvh=kvh, block_size=128, seed=4400 + 16 * group + len(new), poison=True)
    a, b = _run(c), _run(c)
    assert np.array_equal(torch_to_bits(a), torch_to_bits(b))
    assert_attention_close(torch_to_f32(a), _want(c), f"group {group}: {prefixes} + {new}")
    assert _lib.device_status() == 0


@pytest.mark.parametrize("group", [1, 4, 5, 8])
@pytest.mark.parametrize("prefixes,new", [([895, 896, 897], [1, 128, 129]), ([1025, 0], [3, 700]), ([2000], [50])])
def test_runs_of_two_tiles_match_the_oracle(group, prefixes, new):
    from nanovllm_jax_b200 import _lib
    c = _case(prefixes, new, h=group, kvh=1, block_size=256, seed=4700 + group + prefixes[0], poison=True)
    assert_attention_close(torch_to_f32(_run(c)), _want(c), f"group {group}: {prefixes} + {new}")
    assert _lib.device_status() == 0
