"""The workloads that this library's speed is judged by, as a user's program calls it.

One attention layer of a paged-KV serving engine sees five kinds of call, and each is a kind of case here:

  decode    ``Attention.__call__`` on a decode step: store the step's K/V rows, attend over the pages
  step      a whole decode step of a serving loop: ``DecodeMetadata.update`` once, then one ``fused_decode_step`` per
            layer, every layer with a cache of its own
  prefill   ``Attention.__call__`` on packed prompts: store the K/V rows, causal attention over the packed tensors
  prefix    the same when a prefix of every prompt is in the cache already: keys and values come from the pages
  pre       ``qk_norm_rope_store``: the step between the QKV projection and the attention of a prefill batch
  store     ``store_kv_to_cache`` by itself (only drawn: every prefill and decode case contains it)

Not here: the sum over ranks (``PeerAllReduce``), which takes several GPUs.

Sequence lengths are the evenly spaced quantiles of the stated range, so that a case has the same work whatever the
seed; the seed shuffles them over the batch, deals the pages and draws every tensor (N(0, 1) rounded to bf16, as the
activations behind a norm are).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nanovllm_jax_b200 import ops
from nanovllm_jax_b200.layers.attention import Attention, store_kv_to_cache
from nanovllm_jax_b200.utils.context import create_decode_context, create_prefill_context
from nanovllm_jax_b200.utils.decode_metadata import DecodeMetadata, bucket_batch

D = 128
DEVICE = "cuda"
MAX_POSITIONS = 40960  # rows of the rotary table


def _decode(name, batch, heads, kv_heads, lo, hi, log=False, block=256, kv="bf16"):
    return {"name": name, "kind": "decode", "batch": batch, "heads": heads, "kv_heads": kv_heads, "lo": lo, "hi": hi,
            "log": log, "block": block, "kv": kv}


def _prefill(name, batch, heads, kv_heads, lo, hi, block=256, host=True):
    return {"name": name, "kind": "prefill", "batch": batch, "heads": heads, "kv_heads": kv_heads, "lo": lo, "hi": hi,
            "log": False, "block": block, "host": host}


def listed():
    return [
        # one user's chat on the smallest model (16 / 8 heads): the shortest call there is, a layer's latency counts
        _decode("decode-b1-h16", 1, 16, 8, 300, 300),
        # the small configuration: eight conversations of 64 to 1024 tokens
        _decode("decode-b8-h16", 8, 16, 8, 64, 1024),
        # the headline configuration: 64 conversations of 512 to 8192 tokens on 32 / 8 heads
        _decode("decode-b64-h32", 64, 32, 8, 512, 8192),
        # the large configuration: 256 sequences of very different lengths on 64 / 8 heads
        _decode("decode-b256-h64-skewed", 256, 64, 8, 16, 32768, log=True),
        # the same on one rank of eight: each has one kv head
        _decode("decode-b256-h8-shard", 256, 8, 1, 16, 32768, log=True),
        # a step of the serving benchmark: 36 layers, 120 requests (padded to the 128 bucket) with 512 prompt tokens and
        # up to 256 generated ones; host metadata, q/k norm, rotary embedding, store and attention
        {"name": "step-b120-h32-36-layers", "kind": "step", "batch": 120, "heads": 32, "kv_heads": 8, "lo": 513, "hi": 768,
         "log": False, "block": 256, "layers": 36},
        # time to first token of one short prompt on the smallest model
        _prefill("prefill-1x87-h16", 1, 16, 8, 87, 87),
        # a burst of short prompts on a shard with an odd number of query heads per kv head, lengths on the device only
        _prefill("prefill-48-short-h10", 48, 10, 2, 5, 300, host=False),
        # the prefill configuration: 16 prompts of 128 to 4096 tokens on 32 / 8 heads
        _prefill("prefill-16-h32", 16, 32, 8, 128, 4096),
        # one long document, as many tokens as the engine puts into a prefill batch, on 64 / 8 heads
        _prefill("prefill-1x16384-h64", 1, 64, 8, 16384, 16384),
        # a new question behind a cached system prompt or an earlier conversation
        {"name": "prefix-12-h32", "kind": "prefix", "batch": 12, "heads": 32, "kv_heads": 8, "lo": 17, "hi": 700,
         "log": False, "pre_lo": 500, "pre_hi": 5000, "block": 256, "host": True},
        # between projection and attention of a full prefill batch
        {"name": "pre-16384-h32", "kind": "pre", "tokens": 16384, "heads": 32, "kv_heads": 8, "block": 256},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kv_heads = rng.choice((1, 2, 4, 8, 8))
    group = rng.choice((1, 2, 3, 4, 4, 5, 7, 8, 8))
    heads = kv_heads * group
    block = rng.choice((128, 256, 256, 256, 512))
    kind = rng.choice(("decode", "decode", "decode", "step", "prefill", "prefill", "prefill", "prefix", "prefix", "pre",
                       "store"))
    if kind in ("pre", "store"):
        c = {"kind": kind, "tokens": _log_int(rng, 1, 32768), "heads": heads, "kv_heads": kv_heads, "block": block}
        if kind == "store":
            c["kv"] = rng.choice(("bf16", "bf16", "f32"))
        return c
    if kind in ("decode", "step"):
        batch = _log_int(rng, 1, 256)
        layers = rng.randint(2, 36) if kind == "step" else 1
        most = 4.0e9 / (layers * batch * kv_heads * D * 4)  # tokens a sequence, so that the caches stay below 4 GB
        hi = _log_int(rng, 2, int(max(2, min(32768, most))))
        lo = _log_int(rng, 1, hi)
        c = {"kind": kind, "batch": batch, "heads": heads, "kv_heads": kv_heads, "lo": lo, "hi": hi,
             "log": rng.random() < 0.5, "block": block}
        if kind == "decode":
            c["kv"] = rng.choice(("bf16", "bf16", "bf16", "f32"))
        else:
            c["layers"] = layers
        return c
    batch = _log_int(rng, 1, 64)
    hi = _log_int(rng, 2, 16384 if kind == "prefill" else 4096)
    hi = max(2, min(hi, 65536 // batch))
    lo = _log_int(rng, 1, hi)
    c = {"kind": kind, "batch": batch, "heads": heads, "kv_heads": kv_heads, "lo": lo, "hi": hi, "log": False,
         "block": block, "host": rng.random() < 0.7}
    if kind == "prefix":
        c["pre_hi"] = _log_int(rng, 2, min(16384, max(2, 262144 // batch)))
        c["pre_lo"] = rng.randint(1, c["pre_hi"])
    while work(c)["flops"] > 4.0e12:
        c["batch"] = max(1, c["batch"] // 2)
    return c


# ---- lengths, pages, tensors ---------------------------------------------------------------------------------------


def _lengths(n, lo, hi, log):
    at = (np.arange(n) + 0.5) / n
    x = np.exp(math.log(lo) + at * (math.log(hi) - math.log(lo))) if log else lo + at * (hi - lo)
    return np.clip(np.rint(x), lo, hi).astype(np.int64)


def _pages(rng, lens, block, pool):
    """Page ids per sequence and the padded block tables, dealt at random from a pool of ``pool`` pages."""
    need = -(-lens // block)
    perm = rng.permutation(pool).astype(np.int32)
    cut = np.concatenate([[0], np.cumsum(need)])
    lists = [perm[cut[i]:cut[i + 1]].tolist() for i in range(len(lens))]
    tables = np.full((len(lens), int(need.max())), -1, np.int32)
    for i, ids in enumerate(lists):
        tables[i, :len(ids)] = ids
    return lists, tables


def _pool(block, *lens):
    """Pages that hold the lengths (of prefixes and of new tokens, in any pairing), and an eighth more."""
    most = int(sum((-(-x // block)).sum() for x in lens))
    return most + most // 8 + 8


def _slots(lists, first, last, block):
    """Cache slots of tokens first[b] .. last[b] - 1 of every sequence, packed."""
    parts = []
    for ids, a, z in zip(lists, first, last):
        tok = np.arange(a, z)
        parts.append(np.asarray(ids, np.int64)[tok // block] * block + tok % block)
    return np.concatenate(parts).astype(np.int32)


def _normal(gen, shape, dtype=torch.bfloat16):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype)


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEVICE)


def _kv_dtype(case):
    return torch.float32 if case.get("kv") == "f32" else torch.bfloat16


def _rotary_table():
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device=DEVICE, dtype=torch.float32) / D))
    ang = torch.arange(MAX_POSITIONS, device=DEVICE, dtype=torch.float32)[:, None] * inv[None, :]
    return torch.cat([ang.cos(), ang.sin()], dim=-1).contiguous()


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    kind, h, kvh, block = case["kind"], case["heads"], case["kv_heads"], case["block"]
    s = {"kind": kind}

    if kind in ("pre", "store"):
        t = case["tokens"]
        blocks = -(-t // block) + 1
        s["slots"] = _dev(rng.permutation(blocks * block)[:t].astype(np.int32)) if t < 64 else _dev(
            _slots([rng.permutation(blocks).tolist()], [0], [t], block))
        s["k_cache"], s["v_cache"] = (torch.zeros((blocks, block, kvh, D), dtype=torch.bfloat16, device=DEVICE)
                                      for _ in range(2))
        s["k"], s["v"] = (_normal(gen, (t, kvh, D), _kv_dtype(case)) for _ in range(2))
        if kind == "pre":
            s["q"] = _normal(gen, (t, h, D))
            s["q_w"], s["k_w"] = (1.0 + 0.1 * _normal(gen, (D,), torch.float32) for _ in range(2))
            s["table"] = _rotary_table()
            s["positions"] = _dev((np.arange(t) % 16384).astype(np.int32))
        return s

    batch, log = case["batch"], case["log"]
    lens = rng.permutation(_lengths(batch, case["lo"], case["hi"], log))
    attn = s["attn"] = Attention(h, D, 1.0 / math.sqrt(D), kvh, block)

    if kind in ("decode", "step"):
        pool = _pool(block, lens)
        lists, tables = _pages(rng, lens, block, pool)
        slots = _slots(lists, lens - 1, lens, block)
        if kind == "decode":
            attn.set_kv_cache(_normal(gen, (pool, block, kvh, D)), _normal(gen, (pool, block, kvh, D)))
            s["q"] = _normal(gen, (batch, h, D))
            s["k"], s["v"] = (_normal(gen, (batch, kvh, D), _kv_dtype(case)) for _ in range(2))
            s["ctx"] = create_decode_context(_dev(lens.astype(np.int32)), _dev(slots), _dev(tables))
            return s
        layers, rows = case["layers"], bucket_batch(batch, 512)
        s["metadata"] = DecodeMetadata(rows, tables.shape[1], DEVICE)
        s["lists"] = (rng.integers(0, 151936, batch).tolist(), (lens - 1).tolist(), slots.tolist(), lens.tolist(), lists)
        s["k_cache"], s["v_cache"] = (_normal(gen, (layers, pool, block, kvh, D)) for _ in range(2))
        s["q"], s["out"] = _normal(gen, (layers, rows, h, D)), torch.empty((layers, rows, h, D), dtype=torch.bfloat16,
                                                                          device=DEVICE)
        s["k"], s["v"] = (_normal(gen, (layers, rows, kvh, D)) for _ in range(2))
        s["per_layer"] = list(zip(*(x.unbind(0) for x in (s["q"], s["k"], s["v"], s["k_cache"], s["v_cache"], s["out"]))))
        s["q_w"], s["k_w"] = (1.0 + 0.1 * _normal(gen, (D,), torch.float32) for _ in range(2))
        s["table"] = _rotary_table()
        return s

    pre = np.zeros(batch, np.int64)
    if kind == "prefix":
        pre = rng.permutation(_lengths(batch, case["pre_lo"], case["pre_hi"], False))
    pool = _pool(block, pre, lens)
    lists, tables = _pages(rng, pre + lens, block, pool)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cu_k = np.concatenate([[0], np.cumsum(pre + lens)]).astype(np.int32)
    cu_dev = _dev(cu)
    attn.set_kv_cache(_normal(gen, (pool, block, kvh, D)), _normal(gen, (pool, block, kvh, D)))
    t = int(cu[-1])
    s["q"], s["k"], s["v"] = _normal(gen, (t, h, D)), _normal(gen, (t, kvh, D)), _normal(gen, (t, kvh, D))
    s["ctx"] = create_prefill_context(
        cu_dev, _dev(cu_k) if kind == "prefix" else cu_dev, int(lens.max()), int((pre + lens).max()),
        _dev(_slots(lists, pre, pre + lens, block)), block_tables=_dev(tables) if kind == "prefix" else None,
        cu_seqlens_host=cu if case["host"] else None)
    return s


def run(s):
    kind = s["kind"]
    if kind == "store":
        store_kv_to_cache(s["k"], s["v"], s["k_cache"], s["v_cache"], s["slots"])
        return {"k_cache": s["k_cache"], "v_cache": s["v_cache"]}
    if kind == "pre":
        ops.qk_norm_rope_store(s["q"], s["k"], s["v"], s["q_w"], s["k_w"], s["table"], s["positions"], s["k_cache"],
                               s["v_cache"], s["slots"])
        return {"q": s["q"], "k": s["k"], "k_cache": s["k_cache"], "v_cache": s["v_cache"]}
    attn = s["attn"]
    if kind == "step":
        md = s["metadata"]
        md.update(*s["lists"], max_num_seqs=512)
        ctx = md.context()
        ids, positions = md.inputs()
        for q, k, v, k_cache, v_cache, out in s["per_layer"]:
            ops.fused_decode_step(q, k, v, s["q_w"], s["k_w"], s["table"], positions, k_cache, v_cache, ctx.slot_mapping,
                                  ctx.block_tables, ctx.context_lens, attn.scale, attn.block_size, out=out)
        return {"out": s["out"], "q": s["q"], "k": s["k"], "k_cache": s["k_cache"], "v_cache": s["v_cache"], "ids": ids,
                "positions": positions, "slots": ctx.slot_mapping, "lens": ctx.context_lens, "tables": ctx.block_tables}
    out = attn(s["q"], s["k"], s["v"], s["ctx"])
    return {"out": out, "k_cache": attn.k_cache, "v_cache": attn.v_cache}


def work(case):
    kind, h, kvh = case["kind"], case["heads"], case["kv_heads"]
    src = 4 if case.get("kv") == "f32" else 2
    if kind == "store":
        return {"bytes": case["tokens"] * (2 * kvh * D * (src + 2) + 4), "flops": 0}
    if kind == "pre":  # q, k, v read; q, k and the two cache rows written; slot and position; a row of the rotary table
        t = case["tokens"]
        return {"bytes": t * (2 * D * (2 * h + 5 * kvh) + 8) + min(t, 16384) * 4 * D, "flops": 0}
    lens = _lengths(case["batch"], case["lo"], case["hi"], case["log"])
    if kind in ("decode", "step"):
        ctx, b, pages = int(lens.sum()), case["batch"], int((-(-lens // case["block"])).sum())
        # the live cache rows but the newest (which comes from k and v), q, out, and the new rows in and out
        layer = (ctx - b) * kvh * D * 4 + 2 * b * h * D * 2 + 2 * b * kvh * D * (src + 2)
        if kind == "step":
            layer += b * h * D * 2 + b * kvh * D * 2  # q and k are updated in place
        layers = case.get("layers", 1)
        return {"bytes": layers * layer + 4 * (pages + 4 * b), "flops": layers * 4 * ctx * h * D}
    t = int(lens.sum())
    pre = _lengths(case["batch"], case["pre_lo"], case["pre_hi"], False) if kind == "prefix" else np.zeros(1, np.int64)
    # the shuffles pair lengths and prefixes at random: their mean product
    keys = float(lens.sum() * pre.mean() + (lens * (lens + 1) // 2).sum())
    size = t * D * 2 * (2 * h + 4 * kvh) + int(pre.sum()) * kvh * D * 4 + 4 * t
    return {"bytes": size, "flops": 4 * D * h * keys}


def tolerance(case):
    """Data movement and the norm / rotary step (separate IEEE operations in a fixed order) give the same bits; attention
    rounds the probabilities and the result to bf16 (2^-9 each), and sums in an order of its own."""
    return "exact" if case["kind"] in ("pre", "store") else {"rel": 1e-2, "max": 5e-2}
