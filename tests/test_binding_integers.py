"""Integer arguments of the native operators: a size that is not whole is refused as the comparison with the tensor's own
size did, and never cut; ``max_seqlen``, an upper bound only, takes what ``int()`` takes."""
import numpy as np
import pytest


class _Index:
    def __index__(self):
        return 256


def _prefill_step(block_size, heads=4):
    """Reaches the operator's integers with CPU tensors; what is accepted ends at the check that q is on a GPU."""
    import torch
    from nanovllm_jax_b200 import _lib
    bf = dict(dtype=torch.bfloat16)
    q, k, cache = torch.zeros(3, 4, 128, **bf), torch.zeros(3, 2, 128, **bf), torch.zeros(1, 256, 2, 128, **bf)
    i32 = torch.zeros(2, dtype=torch.int32)
    return _lib.binding().prefill_step(q, k, k, cache, cache, i32, None, i32, i32, 16, 0.1, block_size, heads, 2, None)


@pytest.mark.parametrize("bad", [256.5, np.float32(255.9), np.float64(256.25), float("nan"), "256"])
def test_sizes_that_are_not_whole_are_refused(bad):
    with pytest.raises((ValueError, TypeError)) as e:
        _prefill_step(bad)
    assert "CUDA tensor" not in str(e.value), "cut to an integer"


def test_values_of_more_than_32_bits_are_refused():
    for big in (1 << 40, 2.0 ** 40, float("inf")):
        with pytest.raises(OverflowError):
            _prefill_step(big)


@pytest.mark.parametrize("good", [256, 256.0, np.int64(256), np.int32(256), np.float32(256), _Index()])
def test_whole_sizes_of_any_type_are_taken(good):
    with pytest.raises(TypeError, match="q must be a CUDA tensor"):
        _prefill_step(good)


def test_a_tensor_scalar_is_taken():
    import torch
    for good in (torch.tensor(256), torch.tensor(256.0)):
        with pytest.raises(TypeError, match="q must be a CUDA tensor"):
            _prefill_step(good)


def test_another_block_size_is_the_callers_matter():
    assert _prefill_step(128) is None


@pytest.mark.gpu
def test_operators_on_the_gpu():
    import math
    import torch
    from conftest import assert_attention_close, torch_to_f32
    from nanovllm_jax_b200 import ops
    torch.manual_seed(5)
    q, k, v = (torch.randn(40, 2, 128, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    cu = torch.tensor([0, 40], dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(128)
    want = torch.nn.functional.scaled_dot_product_attention(*(x.float().transpose(0, 1) for x in (q, k, v)), is_causal=True,
                                                            scale=scale).transpose(0, 1)
    for longest in (40, 40.7, np.int64(64), "40"):
        assert_attention_close(torch_to_f32(ops.varlen_prefill(q, k, v, cu, longest, scale)), torch_to_f32(want), f"{longest!r}")
    cache = torch.randn(1, 256, 2, 128, dtype=torch.bfloat16, device="cuda")
    tables, lens = torch.zeros(1, 1, dtype=torch.int32, device="cuda"), torch.full((1,), 9, dtype=torch.int32, device="cuda")
    one = ops.paged_decode(q[:1], cache, cache, tables, lens, scale, 256)
    assert torch.equal(one, ops.paged_decode(q[:1], cache, cache, tables, lens, scale, 256.0))
    for bad in (256.5, "256"):
        with pytest.raises((ValueError, TypeError)):
            ops.paged_decode(q[:1], cache, cache, tables, lens, scale, bad)
