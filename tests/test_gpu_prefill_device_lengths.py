"""A prefill follows the lengths in the device's cu_seqlens: the host copy only sizes the grid.  A captured call is replayed
with other lengths than it was captured with (the same number of sequences and packed tokens), among them more token
blocks than the host copy had."""
import numpy as np
import pytest

from conftest import assert_attention_close, bits_to_torch, torch_to_bits, torch_to_f32

pytestmark = pytest.mark.gpu

# kind of launch -> heads, kv heads, lengths at the capture, lengths of the replays
CASES = {
    "short": (8, 2, [87, 40, 0, 131], [[1, 128, 129, 0], [0, 0, 0, 258], [100, 100, 58, 0], [64, 64, 65, 65]]),
    "short, odd group": (3, 1, [300, 5], [[5, 300], [130, 129], [0, 1]]),
    # items cut into runs (eight K/V tiles or more); then more items than runs were foreseen, which stay whole
    "split": (4, 1, [1536] + [0] * 23, [[36, 1500] + [0] * 22, [64] * 24, [0] * 23 + [1024], [100] * 14 + [0] * 10]),
    # four token blocks of 64 at the capture, eight sequences in a replay: several items a CTA
    "short, more items than CTAs": (8, 2, [256] + [0] * 7, [[32] * 8, [1, 3, 250, 2, 0, 0, 0, 0]]),
}


@pytest.mark.parametrize("step", [False, True])
@pytest.mark.parametrize("kind", CASES)
def test_replay_follows_the_device_lengths(kind, step):
    import torch
    from nanovllm_jax_b200 import _lib, ops, workloads
    from nanovllm_jax_b200.layers.attention import Attention
    from nanovllm_jax_b200.utils.context import create_prefill_context
    from oracle import reference_attention as ref
    h, kvh, lens, replays = CASES[kind]
    w = workloads.make_prefill_workload("device-lengths", seed=9700 + len(lens) + h, batch=len(lens), num_heads=h,
                                        num_kv_heads=kvh, len_lo=1, len_hi=1, seq_lens=lens)
    t = workloads.prefill_tensors_numpy(w)
    q, k, v = (bits_to_torch(t[n + "_bits"]) for n in "qkv")
    cu = torch.from_numpy(w.cu_seqlens).cuda()
    slots = torch.arange(w.total_tokens, dtype=torch.int32, device="cuda")
    attn = Attention(h, 128, w.scale, kvh, 256)
    if step:
        attn.set_kv_cache(*(torch.zeros((w.total_tokens // 256 + 1, 256, kvh, 128), dtype=torch.bfloat16, device="cuda")
                            for _ in range(2)))

    def call():
        ctx = create_prefill_context(cu, cu, max(lens), max(lens), slots, cu_seqlens_host=w.cu_seqlens)
        return attn(q, k, v, ctx)

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = call()
    for new in [lens] + replays:
        new_cu = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
        cu.copy_(torch.from_numpy(new_cu))
        if step:
            attn.k_cache.zero_()
        graph.replay()
        torch.cuda.synchronize()
        n = int(new_cu[-1])
        want = ref.variable_length_attention_prefill(t["q"][:n], t["k"][:n], t["v"][:n], new_cu, new_cu, 8192, 8192, h, kvh,
                                                     w.scale, len(new))
        assert_attention_close(torch_to_f32(out)[:n], want, f"{kind}: captured with {lens}, replayed with {new}")
        if step:
            assert np.array_equal(torch_to_bits(attn.k_cache).reshape(-1, kvh, 128)[:w.total_tokens], t["k_bits"])
    assert _lib.device_status() == 0


@pytest.mark.parametrize("h,kvh,lens", [(2, 1, [9300]), (1, 1, [8200, 3]), (2, 1, [300, 8700])])
def test_prompts_beyond_the_contexts_length_bucket(h, kvh, lens):
    """The context's max_seqlen_q ends at 8192, and without a host copy the library sizes its grid from it: prompts beyond it
    have more token blocks than foreseen (with so few heads the launch cuts its items into runs)."""
    import torch
    from nanovllm_jax_b200 import _lib, workloads
    from nanovllm_jax_b200.layers.attention import Attention
    from nanovllm_jax_b200.utils.context import create_prefill_context
    w = workloads.make_prefill_workload("long", seed=9800 + lens[0], batch=len(lens), num_heads=h, num_kv_heads=kvh, len_lo=1,
                                        len_hi=1, seq_lens=lens)
    t = workloads.prefill_tensors_numpy(w)
    q, k, v = (bits_to_torch(t[n + "_bits"]) for n in "qkv")
    cu = torch.from_numpy(w.cu_seqlens).cuda()
    attn = Attention(h, 128, w.scale, kvh, 256)
    ctx = create_prefill_context(cu, cu, max(lens), max(lens), torch.arange(w.total_tokens, dtype=torch.int32, device="cuda"))
    assert ctx.max_seqlen_q == 8192
    got = torch_to_f32(attn(q, k, v, ctx))
    for a, z in zip(w.cu_seqlens[:-1], w.cu_seqlens[1:]):
        s = (q[a:z].float().transpose(0, 1) @ k[a:z].float().permute(1, 2, 0)) * w.scale
        s.masked_fill_(torch.ones(z - a, z - a, dtype=torch.bool, device="cuda").triu_(1), float("-inf"))
        want = (s.softmax(-1) @ v[a:z].float().transpose(0, 1)).transpose(0, 1)
        assert_attention_close(got[a:z], torch_to_f32(want), f"{lens} rows {a}..{z}")
    assert _lib.device_status() == 0
