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

// Many tokens: a warp works on eight rows of one token at a time (a pass), four lanes per row: first the q rows, then the
// k and v rows.  A work unit is `span` consecutive passes of a token; the units are dealt round-robin to a persistent grid.
// The token's cosines and sines are loaded once per unit and stay in registers over its passes, only the eight weight loads
// of a pass come from shared memory, and the rows of the next pass are requested before the current one is computed.
// Bound by instruction latency at 16 warps per SM (16 384 tokens, 32 / 8 heads: 87.2 us with a row per four lanes and the
// rotation loaded for every row, 79.5 us here = 5.6 TB/s; rows staged through shared memory with bulk copies, 142 us).
constexpr int kPassThreads = 256;
__global__ void __launch_bounds__(kPassThreads, 2) pre_attention_pass_kernel(const Params p, const int passes, const int span) {
    __shared__ __align__(16) float weights[2][kD];
    griddep_wait();  // q, k, v may come from the kernel just before this one (the QKV projection)
    griddep_launch_dependents();
    weights[threadIdx.x >> 7][threadIdx.x & 127] = (threadIdx.x < kD ? p.q_weight : p.k_weight - kD)[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, q = lane & 3, sub = lane >> 2;
    const int q_passes = (p.H + 7) >> 3;
    const int parts = (passes + span - 1) / span;  // units per token
    const int64_t units = p.T * parts, stride = (int64_t)gridDim.x * (kPassThreads / 32);

    int64_t unit = (int64_t)blockIdx.x * (kPassThreads / 32) + (threadIdx.x >> 5);
    if (unit >= units) return;
    int64_t t = unit / parts;
    int pass = (int)(unit - t * parts) * span, end = min(pass + span, passes);

    auto source = [&](int64_t tok, int ps) -> const __nv_bfloat16* {  // this lane's row in a pass (null: none)
        if (ps < q_passes) {
            const int r = ps * 8 + sub;
            return r < p.H ? p.q + (tok * p.H + r) * kD : nullptr;
        }
        const int r = (ps - q_passes) * 8 + sub;
        return r < p.KVH ? p.k + (tok * p.KVH + r) * kD : (r < 2 * p.KVH ? p.v + (tok * p.KVH + r - p.KVH) * kD : nullptr);
    };
    auto load = [&](const __nv_bfloat16* src, uint4 (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            w[i] = src ? *reinterpret_cast<const uint4*>(src + (q + 4 * i) * 8) : make_uint4(0, 0, 0, 0);
    };

    auto store = [&](__nv_bfloat16* dst, const uint4 (&w)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(dst + (q + 4 * i) * 8) = w[i];
    };

    const __nv_bfloat16* src = source(t, pass);
    uint4 w[4];
    load(src, w);
    uint64_t c[2][4], s[2][4];
    int64_t slot = -1;
    bool fresh = true;  // t's metadata and rotation are not loaded yet
    while (true) {
        if (fresh) {
            const int pos = __ldg(p.positions + t);
            slot = __ldg(p.slot_mapping + t);
            load_rotation(p, pos, q, c, s);
            fresh = false;
        }
        int64_t next_t = t;
        int next_pass = pass + 1;
        bool more = true;
        const bool new_unit = next_pass == end;
        if (new_unit) {
            unit += stride;
            more = unit < units;
            if (more) {
                next_t = unit / parts;
                next_pass = (int)(unit - next_t * parts) * span;
            }
        }
        const __nv_bfloat16* next_src = more ? source(next_t, next_pass) : nullptr;
        uint4 next_w[4];
        load(next_src, next_w);

        const int r = (pass - q_passes) * 8 + sub;  // row among the k and v rows (negative: a q row)
        const bool is_v = r >= p.KVH;
        const bool cached = src && r >= 0 && slot >= 0 && slot < p.num_slots;
        if (is_v && cached) store(p.v_cache + (slot * p.KVH + r - p.KVH) * kD, w);
        if (!__all_sync(0xffffffffu, is_v || !src)) {
            norm_rope(w, weights[r >= 0] + q * 8, c, s, p.eps, p.one);
            if (src && !is_v) store(const_cast<__nv_bfloat16*>(src), w);  // q and k are updated in place
            if (!is_v && cached) store(p.k_cache + (slot * p.KVH + r) * kD, w);
        }
        if (!more) break;
        fresh = next_t != t;
        if (new_unit) end = min(next_pass + span, passes);
        t = next_t;
        pass = next_pass;
        src = next_src;
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = next_w[i];
    }
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
    // The pass kernel pays where its passes are full and every resident warp (two CTAs per SM) gets ten of them or more.
    const int passes = (H + 7) / 8 + (2 * KVH + 7) / 8;
    const int64_t ctas = 2 * (int64_t)sm_count(), warps = ctas * (preattn::kPassThreads / 32);
    if (T * passes < 10 * warps || 10 * (H + 2 * KVH) < 9 * 8 * passes) {
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
    NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, preattn::pre_attention_pass_kernel, p, passes, span));
    return NVLLM_B200_OK;
}
