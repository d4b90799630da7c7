// Fused pre-attention step, device code: per-head RMSNorm of q and k, rotary embedding, and the scatter of the
// step's K/V rows into the paged cache, in one pass over q, k, v.
//
// Replaces, for one layer (reference models/qwen3.py:157-166):
//     q = q_norm(q); k = k_norm(k)           layers/layernorm.py:31-48  (fp32 math, result cast back to bf16)
//     q, k = rotary_emb(positions, q, k)     layers/rotary_embedding.py:13-37, 97-104  (x1 cos - x2 sin | x2 cos + x1 sin
//                                            in fp32 with the fp32 cos/sin table, halves split at head_dim / 2)
//     store_kv_to_cache(k, v, ...)           layers/attention.py:42-77 (cast to the cache dtype, scatter by slot)
// q and k are updated in place (prefill reads the packed k); k and v rows also go to their cache slots.
//
// HBM-bound: per token (H + 2 KVH) rows of 256 B are read once, the q and k rows written back, the k and v rows
// written to the cache.  Four lanes per row, four 16-byte chunks per lane (chunks q, q+4, q+8, q+12 of the row's sixteen:
// a dim and its rotation partner 64 dims further sit in the same lane, and three quarters of the per-row scalar work --
// the divide and the square root -- that sixteen lanes per row repeated is gone).  The math runs on packed pairs of
// neighbouring dims (.f32x2: two IEEE operations per instruction).
//
// Arithmetic is pinned so that a host restatement reproduces the bf16 results bit for bit: every fp32 operation
// is a separate IEEE round-to-nearest multiply / add / divide / square root (no fused multiply-add, no approximate
// reciprocal square root), and the sum of squares runs in one fixed order: sixteen partial sums of eight elements
// each, left to right, then a butterfly over the sixteen partial sums (index xor 8, 4, 2, 1).
#pragma once

#include "common.cuh"

namespace nvllm {
namespace preattn {

constexpr int kD = 128;
constexpr int kThreads = 64;  // of a block that works row by row: small, so that it fits beside other kernels' CTAs

struct Params {
    __nv_bfloat16* q;
    __nv_bfloat16* k;
    const __nv_bfloat16* v;
    const float* q_weight;
    const float* k_weight;
    const float* cos_sin;      // [max_pos, 128]: cos(64) | sin(64)
    const int32_t* positions;  // [T]
    __nv_bfloat16* k_cache;
    __nv_bfloat16* v_cache;
    const int32_t* slot_mapping;
    int64_t T;
    int H, KVH;
    int64_t num_slots, max_pos;
    float eps;
    float one;  // 1.0f
};

// Packed pairs of fp32: every operation is two separate IEEE round-to-nearest operations.
__device__ __forceinline__ uint64_t pair(float a, float b) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// Sums are written a * one + b, with a `one` (or minus one) that reaches the kernel as an argument: the assembler contracts
// a packed add or subtract behind a packed multiply into one fused operation, explicit rounding or not -- it also sees
// through a constant one -- and the result then differs in the last bit.
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t unpack_bf16(uint32_t u) {
    return pair(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
__device__ __forceinline__ uint32_t pack_pair(uint64_t v) {
    float a, b;
    split(v, a, b);
    return pack_bf16(a, b);
}
// eight consecutive floats as four pairs
__device__ __forceinline__ void load_pairs(const float* src, uint64_t (&f)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = *(reinterpret_cast<const float4*>(src) + 1);
    f[0] = pair(a.x, a.y), f[1] = pair(a.z, a.w), f[2] = pair(b.x, b.y), f[3] = pair(b.z, b.w);
}

inline int64_t blocks_for(int64_t T, int H, int KVH) {
    return (T * (H + 2 * KVH) * 4 + kThreads - 1) / kThreads;
}

// A quarter of one row as a thread holds it between its loads and its math: lane q (0..3) of the row's four lanes owns
// the 16-byte chunks q, q + 4, q + 8 and q + 12 (chunk c = dims 8c .. 8c+7).
struct Part {
    uint4 w[4];    // the four chunks (zeros for a dead row)
    int64_t t;     // token
    int64_t slot;  // cache slot (k and v rows), -1: none
    int pos;       // position of the token
    int r;         // row of the token: [0, H) q heads, [H, H+KVH) k heads, [H+KVH, H+2KVH) v heads
    bool live;
};

// Issues the loads of lane q's part of row `row` (of the T * (H + 2 KVH) rows); nothing here waits for them.
__device__ __forceinline__ Part load_part(int64_t row, const int q, const Params& p) {
    Part c;
    const int rows_per_token = p.H + 2 * p.KVH;
    c.live = row < p.T * rows_per_token;
    c.t = c.live ? row / rows_per_token : 0;
    c.r = c.live ? (int)(row - c.t * rows_per_token) : 0;
    const int kind = c.r < p.H ? 0 : (c.r < p.H + p.KVH ? 1 : 2);
    const int head = kind == 0 ? c.r : (kind == 1 ? c.r - p.H : c.r - p.H - p.KVH);
    const __nv_bfloat16* src = kind == 0 ? p.q + (c.t * p.H + head) * kD
                                          : (kind == 1 ? p.k : p.v) + (c.t * p.KVH + head) * kD;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        c.w[i] = make_uint4(0, 0, 0, 0);
        if (c.live) c.w[i] = *reinterpret_cast<const uint4*>(src + (q + 4 * i) * 8);
    }
    c.slot = c.live && kind != 0 ? (int64_t)__ldg(p.slot_mapping + c.t) : -1;
    c.pos = c.live ? __ldg(p.positions + c.t) : 0;
    return c;
}

// RMSNorm and rotation of one row over its four lanes, in place.  Lane q holds chunks q, q+4, q+8 and q+12 in w; `weight`
// points at dim 8q of the norm's weights, c and s hold the cosines and sines of chunks q and q + 4.  Every lane of the
// warp must call this together (shuffles).
//
// The sum of squares keeps one fixed order whatever the lane layout: sixteen partial sums, one per chunk, each taken
// front to back, then the butterfly p[c] + p[c ^ 8], + [c ^ 4], + [c ^ 2], + [c ^ 1].  With chunks q, q+4, q+8, q+12
// in one lane the first two levels are local and the last two are shuffles over the row's four lanes.
__device__ __forceinline__ void norm_rope(uint4 (&w)[4], const float* weight, const uint64_t (&c)[2][4],
                                          const uint64_t (&s)[2][4], float eps, float one) {
    uint64_t x[4][4];
    float pp[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t u[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[i][e] = unpack_bf16(u[e]);
            float a, b;
            split(x[i][e], a, b);
            ss = e == 0 ? __fmul_rn(a, a) : __fadd_rn(ss, __fmul_rn(a, a));
            ss = __fadd_rn(ss, __fmul_rn(b, b));
        }
        pp[i] = ss;
    }
    float ss = __fadd_rn(__fadd_rn(pp[0], pp[2]), __fadd_rn(pp[1], pp[3]));  // levels c ^ 8 and c ^ 4
    ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 2));                  // level c ^ 2
    ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 1));                  // level c ^ 1
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(ss, 1.0f / kD), eps)));
    const uint64_t inv2 = pair(inv, inv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint64_t ws[4];
        load_pairs(weight + 32 * i, ws);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[i][e] = unpack_bf16(pack_pair(mul2(mul2(x[i][e], inv2), ws[e])));  // the norm returns bf16
    }
    const uint64_t plus = pair(one, one), minus = pair(-one, -one);
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // chunk q + 4i holds dims d < 64, its rotation partner d + 64 is chunk q + 4i + 8
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            lo[e] = pack_pair(fma2(mul2(x[i + 2][e], s[i][e]), minus, mul2(x[i][e], c[i][e])));  // x1 cos - x2 sin
            hi[e] = pack_pair(fma2(mul2(x[i][e], s[i][e]), plus, mul2(x[i + 2][e], c[i][e])));        // x2 cos + x1 sin
        }
        w[i] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        w[i + 2] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
}

// Cosines and sines of chunks q and q + 4 at a position (clamped to the table).
__device__ __forceinline__ void load_rotation(const Params& p, int64_t pos, int q, uint64_t (&c)[2][4], uint64_t (&s)[2][4]) {
    if (pos < 0) pos = 0;
    if (pos >= p.max_pos) pos = p.max_pos - 1;
    const float* cs = p.cos_sin + pos * kD + q * 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        load_pairs(cs + 32 * i, c[i]);
        load_pairs(cs + 32 * i + 64, s[i]);
    }
}

// Norm, rotation and stores of one part.  Every lane of the warp must call this together (full-warp shuffles; the
// eight rows of a warp may be of different kinds): v rows and dead rows simply do not use the result of the math.
__device__ __forceinline__ void finish_part(const Part& ch, const int q, const Params& p) {
    const int kind = ch.r < p.H ? 0 : (ch.r < p.H + p.KVH ? 1 : 2);
    const int head = kind == 0 ? ch.r : (kind == 1 ? ch.r - p.H : ch.r - p.H - p.KVH);
    uint4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = ch.w[i];
    auto store = [&](__nv_bfloat16* dst) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(dst + (q + 4 * i) * 8) = w[i];
    };
    const bool cached = ch.live && kind != 0 && ch.slot >= 0 && ch.slot < p.num_slots;
    if (kind == 2 && cached) store(p.v_cache + (ch.slot * p.KVH + head) * kD);
    // a warp whose eight rows are all v rows (or past the end) has nothing to compute
    if (__all_sync(0xffffffffu, kind == 2 || !ch.live)) return;
    uint64_t c[2][4], s[2][4];
    load_rotation(p, ch.pos, q, c, s);
    norm_rope(w, (kind == 1 ? p.k_weight : p.q_weight) + q * 8, c, s, p.eps, p.one);
    if (ch.live && kind != 2) store(kind == 0 ? p.q + (ch.t * p.H + head) * kD : p.k + (ch.t * p.KVH + head) * kD);
    if (kind == 1 && cached) store(p.k_cache + (ch.slot * p.KVH + head) * kD);
}

// The share of block `block`: kThreads / 4 of the T * (H + 2 KVH) rows, four lanes per row, 64 bytes
// per lane.
__device__ __forceinline__ void pre_attention_block(int64_t block, const Params& p) {
    const int q = threadIdx.x & 3;
    const Part c = load_part((block * kThreads + threadIdx.x) >> 2, q, p);
    finish_part(c, q, p);
}

}  // namespace preattn
}  // namespace nvllm
