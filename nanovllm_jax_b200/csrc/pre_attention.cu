// qk_norm_rope_store: the stand-alone launch of the fused pre-attention step (see pre_attention.cuh); the decode
// step that folds it into its first kernel lives in paged_decode.cu.
#include "pre_attention.cuh"

namespace nvllm {
namespace preattn {

// Few rows: one row per four lanes and nothing else, so that every SM gets some.
__global__ void __launch_bounds__(kThreads) pre_attention_small_kernel(const Params p) {
    griddep_wait();  // q, k, v may come from the kernel just before this one (the QKV projection)
    griddep_launch_dependents();
    pre_attention_block(blockIdx.x, p);
}

// Many tokens: a warp works on eight rows of one token at a time (a pass), four lanes per row: the q rows, the k rows, the v
// rows.  A work unit is `span` consecutive passes of a token; the units are dealt round-robin to a persistent grid.
// The token's cosines and sines stay in registers over its passes, only the eight weight loads of a pass come from shared
// memory.  The rows of the next pass, and with a new unit its rotation, are copied (cp.async) into the warp's part of shared
// memory while the current one is computed: requested into registers, the rows cost sixteen of them, and a unit began with
// the latencies of its position and of its rotation.
// Bound by HBM: 16 384 tokens, 32 / 8 heads, 445 MB: 81.1 us with the next rows in registers, 73.4 here = 6.1 TB/s.  One pass ahead is
// enough: with two (81.5 us) reads and writes of the DRAM are in each other's way.
constexpr int kPassThreads = 256;
constexpr int kPassStages = 2;  // the pass that is computed and the next one
struct PassSmem {  // of a warp
    uint4 rows[kPassStages][4][32];   // chunk i of each lane's row; every lane copies and reads its own
    float rotation[kPassStages][kD];  // of the units in flight (a unit has at least one pass)
};
constexpr int kPassSmemBytes = kPassThreads / 32 * (int)sizeof(PassSmem);
static_assert(kPassSmemBytes + 2 * kD * 4 <= 48 * 1024, "more than a launch gets without asking");

__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__global__ void __launch_bounds__(kPassThreads, 2) pre_attention_pass_kernel(const Params p, const int passes, const int span) {
    extern __shared__ __align__(16) uint8_t pass_smem[];
    __shared__ __align__(16) float weights[2][kD];
    griddep_wait();  // q, k, v may come from the kernel just before this one (the QKV projection)
    griddep_launch_dependents();
    for (int i = threadIdx.x; i < 2 * kD; i += kPassThreads) weights[i >> 7][i & 127] = (i < kD ? p.q_weight : p.k_weight - kD)[i];
    __syncthreads();
    PassSmem& sm = reinterpret_cast<PassSmem*>(pass_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, q = lane & 3, sub = lane >> 2;
    const int parts = (passes + span - 1) / span;  // units per token
    // a warp's units: the first, and the step to the next one in tokens and parts
    const int warps = gridDim.x * (kPassThreads / 32), step_t = warps / parts, step_part = warps - step_t * parts;

    auto source = [&](int64_t tok, int ps) -> const __nv_bfloat16* {  // this lane's row in a pass (null: none)
        const int r = ps * 8 + sub - p.H;
        if (r < 0) return p.q + (tok * p.H + r + p.H) * kD;
        return r < p.KVH ? p.k + (tok * p.KVH + r) * kD : (r < 2 * p.KVH ? p.v + (tok * p.KVH + r - p.KVH) * kD : nullptr);
    };
    auto store = [&](__nv_bfloat16* dst, const uint4 (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(dst + (q + 4 * i) * 8) = w[i];
    };
    struct Cursor {  // a pass of a unit
        int64_t t;
        int part, pass, end;
    };
    auto enter = [&](Cursor& c) {  // the first pass of its unit
        c.pass = c.part * span;
        c.end = min(c.pass + span, passes);
    };
    auto step = [&](Cursor& c) {  // to the next unit
        c.t += step_t;
        c.part += step_part;
        if (c.part >= parts) c.part -= parts, ++c.t;
        enter(c);
    };

    Cursor at, ahead;
    {
        const int unit = blockIdx.x * (kPassThreads / 32) + (threadIdx.x >> 5);
        at.t = unit / parts;
        at.part = unit - (int)at.t * parts;
    }
    if (at.t >= p.T) return;
    enter(at);
    ahead = at;
    uint32_t filled = 0, entered = 0;  // passes and units copied so far
    int pos = __ldg(p.positions + ahead.t);
    bool fresh_ahead = true;  // ahead's rotation is not on its way yet
    auto fetch = [&]() {  // copies the pass at `ahead` and moves on; one group per call
        if (ahead.t < p.T) {
            if (fresh_ahead) {
                const int64_t row = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
                copy16_async(sm.rotation[entered] + lane * 4, p.cos_sin + row * kD + lane * 4);
                if (++entered == kPassStages) entered = 0;
                Cursor next = ahead;
                step(next);
                if (next.t < p.T) pos = __ldg(p.positions + next.t);
            }
            const __nv_bfloat16* src = source(ahead.t, ahead.pass);
            if (src) {
#pragma unroll
                for (int i = 0; i < 4; ++i) copy16_async(&sm.rows[filled][i][lane], src + (q + 4 * i) * 8);
            }
            if (++filled == kPassStages) filled = 0;
            fresh_ahead = ++ahead.pass == ahead.end;
            if (fresh_ahead) step(ahead);
        }
        copy_commit();
    };
#pragma unroll 1
    for (int i = 0; i + 1 < kPassStages; ++i) fetch();

    uint64_t c[2][4], s[2][4];
    int64_t slot = -1;
    bool fresh = true;  // at's slot and rotation are not loaded yet
    uint32_t done = 0, unit_no = 0;
#pragma unroll 1
    while (true) {
        copy_wait<kPassStages - 2>();
        __syncwarp();  // the other lanes' parts of the rotation; and all have read the buffers that fetch() fills next
        if (fresh) {
            slot = __ldg(p.slot_mapping + at.t);
            const float* cs = sm.rotation[unit_no] + q * 8;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                load_pairs(cs + 32 * i, c[i]);
                load_pairs(cs + 32 * i + 64, s[i]);
            }
            if (++unit_no == kPassStages) unit_no = 0;
        }
        uint4 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = sm.rows[done][i][lane];
        if (++done == kPassStages) done = 0;
        fetch();

        const __nv_bfloat16* src = source(at.t, at.pass);
        const int r = at.pass * 8 + sub - p.H;  // row among the k and v rows (negative: a q row)
        const bool is_v = r >= p.KVH;
        const bool cached = src && r >= 0 && slot >= 0 && slot < p.num_slots;
        if (is_v && cached) store(p.v_cache + (slot * p.KVH + r - p.KVH) * kD, w);
        if (!__all_sync(0xffffffffu, is_v || !src)) {
            norm_rope(w, weights[r >= 0] + q * 8, c, s, p.eps, p.one);
            if (src && !is_v) store(const_cast<__nv_bfloat16*>(src), w);  // q and k are updated in place
            if (!is_v && cached) store(p.k_cache + (slot * p.KVH + r) * kD, w);
        }
        fresh = ++at.pass == at.end;
        if (fresh) {
            step(at);
            if (at.t >= p.T) break;
        }
    }
    copy_wait<0>();
}

int check_args(const char* who, const void* q, const void* k, const void* v, const float* q_weight, const float* k_weight,
               const float* cos_sin_cache, const int32_t* positions, const void* k_cache, const void* v_cache,
               const int32_t* slot_mapping, int64_t T, int H, int KVH, int D, int64_t num_slots, int64_t max_pos) {
    if (T < 0 || H <= 0 || KVH <= 0 || num_slots < 0 || max_pos <= 0)
        return fail(NVLLM_B200_EINVAL, "%s: bad size (T=%lld H=%d KVH=%d num_slots=%lld max_pos=%lld)", who, (long long)T,
                    H, KVH, (long long)num_slots, (long long)max_pos);
    if (D != kD) return fail(NVLLM_B200_EUNSUPPORTED, "%s: head_dim %d (only 128)", who, D);
    if (T == 0) return NVLLM_B200_OK;
    if (!q || !k || !v || !q_weight || !k_weight || !cos_sin_cache || !positions || !k_cache || !v_cache || !slot_mapping)
        return fail(NVLLM_B200_EINVAL, "%s: null pointer", who);
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)q_weight |
         (uintptr_t)k_weight | (uintptr_t)cos_sin_cache) & 15)
        return fail(NVLLM_B200_EINVAL, "%s: buffers must be 16-byte aligned", who);
    if (T * (H + 2 * KVH) > (0x3fffffffLL << 6)) return fail(NVLLM_B200_EUNSUPPORTED, "%s: too many rows", who);
    return NVLLM_B200_OK;
}

}  // namespace preattn
}  // namespace nvllm

extern "C" int nvllm_b200_qk_norm_rope_store(void* q, void* k, const void* v, const float* q_weight, const float* k_weight,
                                             const float* cos_sin_cache, const int32_t* positions, void* k_cache,
                                             void* v_cache, const int32_t* slot_mapping, int64_t T, int H, int KVH, int D,
                                             int64_t num_slots, int64_t max_pos, float eps, void* stream) {
    using namespace nvllm;
    int rc = preattn::check_args("qk_norm_rope_store", q, k, v, q_weight, k_weight, cos_sin_cache, positions, k_cache,
                                 v_cache, slot_mapping, T, H, KVH, D, num_slots, max_pos);
    if (rc || T == 0) return rc;
    preattn::Params p{(__nv_bfloat16*)q, (__nv_bfloat16*)k, (const __nv_bfloat16*)v, q_weight, k_weight, cos_sin_cache,
                      positions, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, slot_mapping, T, H, KVH, num_slots,
                      max_pos, eps, 1.0f};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = reinterpret_cast<cudaStream_t>(stream);
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    // The pass kernel pays where its passes are full and every resident warp (two CTAs per SM) gets 4.5 of them or more (32 / 8 heads,
    // small kernel / this one: 4.1 passes a warp 9.0 / 9.8 us, 5.1 12.7 / 11.5), or eight with passes three quarters full (12 / 4:
    // 5.1 11.1 / 11.5, 7.6 17.4 / 17.0), but not where that is a token's only pass, which loads a rotation every time (4 / 1: 8.4
    // 18.8 / 22.8).
    const int passes = (H + 2 * KVH + 7) / 8;
    const int64_t ctas = 2 * (int64_t)sm_count(), warps = ctas * (preattn::kPassThreads / 32);
    const int rows = H + 2 * KVH, room = 8 * passes;
    const bool many = 10 * rows >= 9 * room ? 2 * T * passes >= 9 * warps
                                            : passes > 1 && 4 * rows >= 3 * room && T * passes >= 8 * warps;
    if (!many) {
        cfg.gridDim = dim3((unsigned)preattn::blocks_for(T, H, KVH));
        cfg.blockDim = dim3(preattn::kThreads);
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, preattn::pre_attention_small_kernel, p));
        return NVLLM_B200_OK;
    }
    // Passes per unit: long units load fewer rotations (about half a pass each), short ones leave a shorter last round.
    int span = 1;
    double best = 0;
    for (int s = 1; s <= passes; ++s) {
        const int64_t units = T * ((passes + s - 1) / s);
        const double cost = (double)((units + warps - 1) / warps) * (s + 0.5);
        if (s == 1 || cost < best) best = cost, span = s;
    }
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(preattn::kPassThreads);
    cfg.dynamicSmemBytes = preattn::kPassSmemBytes;
    NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, preattn::pre_attention_pass_kernel, p, passes, span));
    return NVLLM_B200_OK;
}
