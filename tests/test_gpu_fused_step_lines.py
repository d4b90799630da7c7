"""fused_decode_step around the batch from which its producers request a ring of tiles ahead of q instead of one (as many
sequences as the launch has chunks), with sequences of one tile, of a few and of many, against the separate calls bit for bit."""
import numpy as np
import pytest

from conftest import torch_to_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,kvh", [(8, 1), (20, 4), (64, 8)])
@pytest.mark.parametrize("off", [-1, 0, 1])
@pytest.mark.parametrize("hi", [40, 400, 1500])
def test_equals_the_separate_calls(h, kvh, off, hi):
    import torch
    from nanovllm_jax_b200 import _lib, ops
    batch = 2 * torch.cuda.get_device_properties(0).multi_processor_count // kvh + off
    rng = np.random.Generator(np.random.PCG64(6300 + h + off + hi))
    gen = torch.Generator(device="cuda").manual_seed(6300 + h + off + hi)
    ctx = rng.integers(1, hi + 1, batch)
    need = -(-ctx // 256)
    pages = rng.permutation(int(need.sum()))
    tables = np.full((batch, int(need.max())), -1, np.int32)
    for b, at in enumerate(np.concatenate([[0], np.cumsum(need)[:-1]])):
        tables[b, :need[b]] = pages[at:at + need[b]]
    slots = tables[np.arange(batch), (ctx - 1) // 256] * 256 + (ctx - 1) % 256
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.int32)).cuda()
    normal = lambda *shape, dtype=torch.bfloat16: torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    sl, bt, cl, pos = dev(slots), dev(tables), dev(ctx), dev(ctx - 1)
    q, k, v = normal(batch, h, 128), normal(batch, kvh, 128), normal(batch, kvh, 128)
    kc, vc = (normal(len(pages), 256, kvh, 128) for _ in range(2))
    args = (*(1 + 0.1 * normal(128, dtype=torch.float32) for _ in range(2)), normal(2048, 128, dtype=torch.float32), pos)
    q1, k1, kc1, vc1 = q.clone(), k.clone(), kc.clone(), vc.clone()
    ops.qk_norm_rope_store(q1, k1, v, *args, kc1, vc1, sl)
    want = ops.paged_decode(q1, kc1, vc1, bt, cl, 128 ** -0.5, 256)
    for _ in range(3):  # back to back, as the layers of a step
        q2, k2, kc2, vc2 = q.clone(), k.clone(), kc.clone(), vc.clone()
        got = ops.fused_decode_step(q2, k2, v, *args, kc2, vc2, sl, bt, cl, 128 ** -0.5, 256)
        for x, y in ((got, want), (q2, q1), (k2, k1), (kc2, kc1), (vc2, vc1)):
            assert np.array_equal(torch_to_bits(x), torch_to_bits(y))
    assert _lib.device_status() == 0
