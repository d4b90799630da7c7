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


def test_replay_with_more_token_blocks_than_foreseen():
    """A captured call whose items are runs of one tile, replayed with lengths that make more of them than it has CTAs: they stay
    whole, and a CTA takes several."""
    import torch
    from conftest import bits_to_torch
    from nanovllm_jax_b200 import _lib, ops
    h, prefixes = 8, [2600, 1500, 130, 900, 1024, 0, 2000, 64]
    first, replays = [200] + [0] * 7, [[25] * 8, [0, 100, 1, 33, 0, 32, 2, 32], [1, 0, 0, 0, 0, 0, 0, 199]]
    cases = [_case(prefixes, new, h=h, kvh=1, block_size=256, seed=6250) for new in [first] + replays]
    mb, nb = max(c["tables"].shape[1] for c in cases), max(len(c["k_bits"]) for c in cases)
    grow = lambda x: np.pad(x, ((0, nb - len(x)),) + ((0, 0),) * (x.ndim - 1))
    c = cases[0]
    q = bits_to_torch(c["q_bits"])
    kc, vc = (torch.zeros((nb, 256, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    tables = torch.full((8, mb), -1, dtype=torch.int32, device="cuda")
    cu_q, cu_k = (torch.zeros(9, dtype=torch.int32, device="cuda") for _ in range(2))
    out = torch.empty_like(q)

    def load(c):
        q.copy_(bits_to_torch(c["q_bits"])), kc.copy_(bits_to_torch(grow(c["k_bits"]))), vc.copy_(bits_to_torch(grow(c["v_bits"])))
        tables.copy_(torch.from_numpy(np.pad(c["tables"], ((0, 0), (0, mb - c["tables"].shape[1])), constant_values=-1)))
        cu_q.copy_(torch.from_numpy(c["cu_q"])), cu_k.copy_(torch.from_numpy(c["cu_k"]))

    def call():
        ops.paged_prefill(q, kc, vc, tables, cu_q, cu_k, 200, c["scale"], 256, cu_seqlens_host=c["cu_q"], out=out)

    load(c)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    for x in cases:
        load(x)
        graph.replay()
        torch.cuda.synchronize()
        assert_attention_close(torch_to_f32(out), _want(x), f"{prefixes}, replayed with {np.diff(x['cu_q'])}")
    assert _lib.device_status() == 0
