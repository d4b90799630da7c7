"""The plan kernel on both sides of the batch sizes where it reads the lengths another way (33 and 1024 sequences: a warp takes
several of them, they no longer fit its shared memory) and where its warps stop taking a sequence each (257)."""
import numpy as np
import pytest

from conftest import assert_attention_close, torch_to_f32
from test_gpu_paged_prefill import _case, _run, _want

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [31, 32, 33, 256, 257, 1023, 1024, 1100])
def test_batches_match_the_oracle(batch):
    from nanovllm_jax_b200 import _lib
    rng = np.random.Generator(np.random.PCG64(9100 + batch))
    new = [int(x) for x in rng.integers(1, 12, batch)]
    prefixes = [int(x) for x in rng.integers(0, 9, batch)]
    new[batch // 2], prefixes[batch // 3] = 300, 140
    c = _case(prefixes, new, h=2, kvh=1, block_size=128, seed=9200 + batch, poison=True)
    assert_attention_close(torch_to_f32(_run(c)), _want(c), f"batch {batch}")
    assert _lib.device_status() == 0
