// paged_decode: flash-decoding over the block-table KV cache for sm_100a.
//
// Replaces paged_attention / paged_decode_attention_vectorized of the
// reference (layers/pallas_attention.py:465-507, :146-238).
//
// The op is HBM-bound: every live K and V row is read exactly once.  Design:
//
//  * Work unit = one 64-token tile of one (sequence, kv head).  All tiles of
//    one kv head are laid end to end (sequence after sequence) and cut into
//    `num_groups` contiguous chunks of equal COST ("stream-K" partition): a tile
//    costs one unit and every sequence three more in front of its tiles (the
//    time a CTA loses at a sequence boundary -- q load, page lookup, the
//    cross-warp combine, and the partial results at the ends of a chunk).  So every CTA
//    finishes at the same time no matter how skewed the context lengths are or
//    how many short sequences fall into its chunk.  CTA c serves kv head c % KVH of chunk c / KVH; the KVH CTAs of a
//    chunk walk the same tokens at the same pace, so the 256-byte per-head rows
//    they fetch are neighbours in DRAM.  Small batches use fewer, longer chunks (make_cut).
//  * Persistent CTAs, 2 per SM: one producer warp issues TMA tile loads
//    (cp.async.bulk.tensor, 128-byte swizzle, no multicast, one load per 16 KB tile) into a ring of two
//    or three stages (ring_stages) and runs ahead across sequence boundaries; what a tile is (live tokens, first or last
//    of its sequence, where its result goes) travels beside it in the ring, so only the producer walks the
//    sequences.  Four consumer warps each own 16 tokens of a tile.
//  * The G = H/KVH query heads that share a kv head are the 8 columns of
//    mma.sync.m16n8k16 (bf16 in, fp32 accumulate), tokens and dims its 16 rows: S^T = K Q^T, O^T += V^T P^T (the heads as
//    half-empty rows took twice the instructions and cost 3-5 % of the whole kernel).  The online softmax (exp2
//    domain) lives in registers; the running maximum may be stale by 2^8, so the lanes vote on it instead of
//    reducing it for every tile.
//  * A chunk that ends inside a sequence leaves an fp32 partial (m, l, O) in
//    the caller's workspace and takes a ticket for that (sequence, kv head); the
//    CTA that draws the last ticket combines all partials of the sequence, in
//    chunk order (bitwise reproducible whichever CTA arrives last), and writes
//    the rows -- all G rows at once, every load of a batch of four partials in
//    flight together, so the combine costs about one round trip to L2 per four
//    partials.  Nobody waits for another CTA.  Sequences wholly inside one chunk are
//    written directly.  The tickets are cleared by the small kernel that runs
//    before this one (decode_prepare_kernel, which in the fused decode step
//    also scatters the step's new K/V rows into the cache).
//  * The first tiles are requested before that kernel has finished, unless they hold a slot that it writes.
//
// Measured on a B200 through the decode step (this kernel and the one in front of it, calls in a row, before -> after the
// transposed products, the two-stage ring, the early requests and the native walk): one sequence of 300 tokens, 16 / 8
// heads, 25.0 -> 8.0 us (12.6 -> 7.3 replayed from a graph, where the host's part does not count); Qwen3-8B shapes, batch 64,
// 1.14 GB: 179 -> 168 us (6.8 TB/s); Qwen3-32B shapes, batch 256, 4.51 GB: 673 -> 640 us (7.05 TB/s; 4.5 to 5 %).  What
// bounds it: the stream itself runs at about 7.25 TB/s (a build without the math is not faster); about 3.5 us pass before
// the first tile is under way and 3.5 us after the last one has landed.
//
// No spin-wait is unbounded: every mbarrier wait gives up after a poll limit,
// raises a device error flag (readable through nvllm_b200_device_status) and
// the CTA drains and returns.
#include "pre_attention.cuh"
#include "store_kvcache.cuh"

#include <mutex>
#include <stdlib.h>
#include <string.h>

namespace nvllm {
namespace decode {

constexpr int kTile = 64;                      // tokens per tile
constexpr int kD = 128;                        // head_dim
constexpr int kConsumerWarps = 4;
constexpr int kWarps = kConsumerWarps + 1;     // consumers, TMA producer
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 3;                     // ring stages; long streams use two of them (see ring_stages)
constexpr int kMaxG = 8;                       // query heads per kv head packed in one CTA
constexpr int kItemCostDefault = 3;            // cost of a sequence boundary in tile units (stream-K weights)
constexpr int kPanelBytes = kTile * 128;       // 64 tokens x 64 dims bf16, 128B-swizzled
constexpr int kTileBytes = 2 * kPanelBytes;    // one K or V tile
constexpr int kQBytes = kMaxG * kD * 2;        // 2 KiB
constexpr int kStageBytes = 2 * kTileBytes + kQBytes;  // 34816
constexpr int kOsStride = kD + 4;              // padded row of the cross-warp merge buffers (bank spread)
constexpr int kOsBytes = 2 * kMaxG * kOsStride * 4;  // two buffers [8][132] fp32
constexpr int kMiscBytes = 768 + kThreads * 8;
constexpr int kSmemBytes = kStages * kStageBytes + kOsBytes + kMiscBytes;
static_assert(kSmemBytes + 1024 <= 228 * 1024 / 2, "two CTAs per SM");
constexpr int kCtasPerSm = 2;
constexpr float kStale = 8.f;                  // log2 units by which scores may exceed the running maximum
constexpr int kMergeBatch = 4;                 // partial results the combine has in flight
constexpr int kEarlySlots = 8;                 // slots per producer lane: batches up to 256 request tiles ahead of the wait

// Per-partial record in the workspace: O[G][128] fp32, then m[8], l[8].
__host__ __device__ inline size_t partial_floats(int G) { return (size_t)G * kD + 2 * kMaxG; }

__device__ int g_error_flag = 0;

struct Params {
    const __nv_bfloat16* q;
    const int32_t* block_tables;
    const int32_t* context_lens;
    const int32_t* slot_mapping;  // [B] slots that the kernel just before this one writes, or null: it writes none
    int q_in_flight;              // that kernel writes q too: tiles requested ahead of the wait for it (0: it does not)
    __nv_bfloat16* out;
    float* partials;        // [chunks][KVH][2][partial_floats]
    unsigned int* tickets;  // [B*KVH] partials delivered so far per (sequence, kv head); zero when the kernel starts
    int B, H, KVH, G, NB, block_size, MB;
    int num_groups;
    int item_cost;  // units a sequence boundary costs on the cost line (see units_of)
    float scale_log2;
};

__device__ __forceinline__ int clamp_ctx(int c, int max_ctx) { return c < 0 ? 0 : (c > max_ctx ? max_ctx : c); }
__device__ __forceinline__ int tiles_of(int ctx) { return (ctx + kTile - 1) / kTile; }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

// ------------------------------------------------------------------------------------------
// the cut of the work
// ------------------------------------------------------------------------------------------
// The cost line: sequence b with tb > 0 tiles occupies tb + item_cost units, the first item_cost of them standing
// for its boundary overhead, the rest for its tiles 0 .. tb-1; empty sequences occupy nothing.
__device__ __forceinline__ int units_of(int tb, int item_cost) { return tb > 0 ? tb + item_cost : 0; }

// The line of one kv head (`total` units) is cut into `groups` contiguous chunks, one per CTA: the first `rem` of
// `len + 1` units, the others of `len`.  The cut depends on the lengths alone: the results are bitwise reproducible.
// (Handing the last eighth of the line out dynamically in ever smaller chunks was measured: the CTAs then finish
// together, but at the same time as before -- the stream is bound by DRAM, not by its slowest CTA -- and the many small
// partial results of a long sequence cost up to 15 us to combine.)
struct Cut {
    int groups;
    long long len, rem;

    __device__ __forceinline__ long long bound(int chunk) const { return chunk * len + (chunk < rem ? chunk : rem); }
    // chunk that holds unit u
    __device__ __forceinline__ int chunk_of(long long u) const {
        const long long head = rem * (len + 1);
        return u < head ? (int)div(u, len + 1) : (int)(rem + div(u - head, len));
    }
    // 64-bit divisions are slow and only lines of more than 2^31 units need them
    static __device__ __forceinline__ long long div(long long a, long long b) {
        return ((a | b) >> 31) == 0 ? (long long)((uint32_t)a / (uint32_t)b) : a / b;
    }
};

// Less than kMinChunk units per CTA: chunks of kMinChunk units and fewer CTAs.  Five tiles take about as long as splitting
// them further would cost (partial, ticket, combine: 2.5 us).
constexpr int kMinChunk = 5;
__device__ __forceinline__ Cut make_cut(long long total, int num_groups) {
    Cut c;
    c.groups = num_groups;
    if (total < (long long)kMinChunk * num_groups) c.groups = max(1, (int)total / kMinChunk);
    c.len = Cut::div(total, c.groups);
    c.rem = total - c.len * c.groups;
    return c;
}

// Stages of the ring in use.  A short chunk wants its first tiles requested at once; a long stream is faster with less in
// flight: 128 KB per SM keep DRAM busy, and with 192 KB the requests of all SMs get in each other's way (Qwen3-32B
// shapes, batch 256: 664 us with three stages, 640 with two).
__device__ __forceinline__ uint32_t ring_stages(const Cut& cut) { return cut.len > 16 ? 2u : 3u; }

struct Walk {
    int b;             // next sequence to look at
    long long fv;      // unit at which sequence b starts
    long long x0, x1;  // the chunk's range of units
};
struct Item {
    int b, t0, n;      // sequence, first tile and number of tiles this chunk holds of it
    int ctx, tb;       // its context length and total tiles
    long long fv;      // unit at which the sequence starts (its tile 0 sits at fv + item_cost)
};

// Advance to the next sequence of which the chunk holds at least one tile; false when the chunk is exhausted.
// (hint_b, hint_ctx): a context length the caller has fetched ahead of time (hint_b < 0: none).
__device__ __forceinline__ bool next_item(Walk& w, const Params& p, int max_ctx, Item& it, int hint_b, int hint_ctx) {
    while (w.b < p.B && w.fv < w.x1) {
        const int ctx = clamp_ctx(w.b == hint_b ? hint_ctx : __ldg(p.context_lens + w.b), max_ctx);
        const int tb = tiles_of(ctx);
        const long long t_base = w.fv + p.item_cost;  // unit of tile 0
        it.b = w.b;
        it.fv = w.fv;
        ++w.b;
        w.fv += units_of(tb, p.item_cost);
        if (tb == 0) continue;
        const long long lo = w.x0 - t_base, hi = w.x1 - t_base;
        const int t0 = (int)(lo < 0 ? 0 : (lo > tb ? tb : lo));
        const int t1 = (int)(hi < 0 ? 0 : (hi > tb ? tb : hi));
        if (t0 >= t1) continue;  // only boundary units of this sequence fall into the chunk
        it.t0 = t0;
        it.n = t1 - t0;
        it.ctx = ctx;
        it.tb = tb;
        return true;
    }
    return false;
}

// What the producer tells the consumers about a tile, beside the tile in the ring.
struct TileMeta {
    int valid;   // live tokens from this tile's first token on
    int flags;   // kFirst | kLast | kWhole | kDone
    int b;       // sequence
    int part;    // record of the partial result (an item that is not a whole sequence)
    int gf, gl;  // first and last chunk that hold tiles of the sequence
    int pad[2];
};
constexpr int kFirst = 1, kLast = 2, kWhole = 4, kDone = 8;

// Combine the partials of sequence b (chunks gf .. gl) for kv head kvh and write its G output rows.  Called by the 128
// consumer threads: thread t owns row t / 16 and dims 8 (t % 16) .. 8 (t % 16) + 7.  Partials are taken in chunk order,
// kMergeBatch at a time (all loads of a batch are in flight together), so the result does not depend on which CTA runs this.
__device__ __forceinline__ void merge_sequence(const Params& p, int b, int kvh, int gf, int gl, int ctid) {
    const int r = ctid >> 4, c8 = (ctid & 15) * 8;
    if (r >= p.G) return;
    const size_t pf = partial_floats(p.G);
    float mt = -INFINITY, lt = 0.f;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int g0 = gf; g0 <= gl; g0 += kMergeBatch) {
        float mv[kMergeBatch], lv[kMergeBatch];
        float4 oa[kMergeBatch], ob[kMergeBatch];
#pragma unroll
        for (int u = 0; u < kMergeBatch; ++u) {
            const int g = g0 + u;
            const bool live = g <= gl;
            const float* part = p.partials + ((size_t)(g * p.KVH + kvh) * 2 + (g == gf ? 1 : 0)) * pf;
            mv[u] = live ? __ldcg(part + p.G * kD + r) : -INFINITY;
            lv[u] = live ? __ldcg(part + p.G * kD + kMaxG + r) : 0.f;
            oa[u] = live ? __ldcg(reinterpret_cast<const float4*>(part + r * kD + c8)) : make_float4(0.f, 0.f, 0.f, 0.f);
            ob[u] = live ? __ldcg(reinterpret_cast<const float4*>(part + r * kD + c8) + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float mnew = mt;
#pragma unroll
        for (int u = 0; u < kMergeBatch; ++u) mnew = fmaxf(mnew, mv[u]);
        if (mnew == -INFINITY) continue;
        const float sc = (mt == -INFINITY) ? 0.f : fast_exp2(mt - mnew);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= sc;
        lt *= sc;
#pragma unroll
        for (int u = 0; u < kMergeBatch; ++u) {
            const float f = (mv[u] == -INFINITY) ? 0.f : fast_exp2(mv[u] - mnew);
            acc[0] += oa[u].x * f;
            acc[1] += oa[u].y * f;
            acc[2] += oa[u].z * f;
            acc[3] += oa[u].w * f;
            acc[4] += ob[u].x * f;
            acc[5] += ob[u].y * f;
            acc[6] += ob[u].z * f;
            acc[7] += ob[u].w * f;
            lt += lv[u] * f;
        }
        mt = mnew;
    }
    const float inv = 1.0f / (lt + 1e-9f);
    uint4 w;
    w.x = pack_bf16(acc[0] * inv, acc[1] * inv);
    w.y = pack_bf16(acc[2] * inv, acc[3] * inv);
    w.z = pack_bf16(acc[4] * inv, acc[5] * inv);
    w.w = pack_bf16(acc[6] * inv, acc[7] * inv);
    *reinterpret_cast<uint4*>(p.out + ((size_t)b * p.H + (size_t)kvh * p.G + r) * kD + c8) = w;
}

__device__ __forceinline__ unsigned int atomic_add_acq_rel(unsigned int* addr, unsigned int v) {
    unsigned int old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(addr), "r"(v) : "memory");
    return old;
}

__device__ __forceinline__ bool wait_or_abort(volatile int* abort, uint64_t* bar, uint32_t parity) {
    return mbar_try_wait(bar, parity) || (!*abort && mbar_wait(bar, parity));
}

// The G query rows of (sequence b, kv head kvh), behind the tile in its ring stage.
__device__ __forceinline__ void load_q(const Params& p, uint8_t* stage, uint64_t* bar, int b, int kvh) {
    bulk_load(stage + 2 * kTileBytes, p.q + ((size_t)b * p.H + (size_t)kvh * p.G) * kD, (uint32_t)p.G * kD * 2, bar);
}

// Two CTAs fit an SM (shared memory).  The registers of a third are left free: the blocks of the kernel behind this one on
// the stream (128 or 256 threads) then start, and wait, beside this kernel's CTAs instead of after them, and this kernel's
// CTAs beside the blocks of the kernel in front.
__global__ void __launch_bounds__(kThreads, kCtasPerSm + 1)
paged_decode_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                    const Params p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    float* Os = reinterpret_cast<float*>(smem + kStages * kStageBytes);
    uint8_t* misc = smem + kStages * kStageBytes + kOsBytes;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(misc);            // [kStages]
    uint64_t* empty_bar = full_bar + kStages;                          // [kStages]
    int* sm_i = reinterpret_cast<int*>(misc + 64);                     // scan scratch [8], ticket [1], abort [1]
    volatile int* sm_abort = sm_i + 12;
    float* sm_ml = reinterpret_cast<float*>(misc + 128);               // [2 parities][m|l][4 warps][8 rows]
    TileMeta* sm_meta = reinterpret_cast<TileMeta*>(misc + 640);       // [kStages]
    long long* sm_seg = reinterpret_cast<long long*>(misc + 768);      // [kThreads] unit at which a thread's sequences start

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x % p.KVH;
    const int chunk = blockIdx.x / p.KVH;
    const int max_ctx = p.MB * p.block_size;

    if (smem_u32(smem) & 1023) {  // the swizzled tiles need it; the alignment above asks for it
        if (tid == 0) atomicOr(&g_error_flag, 1);
        griddep_wait();
        return;
    }
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar + s, 1);
            mbar_init(empty_bar + s, kConsumerWarps);
        }
        fence_mbar_init();
        *sm_abort = 0;
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }

    griddep_launch_dependents();  // lets the next kernel of the stream run its own prologue while this grid streams

    // Programmatic dependent launch: this grid starts while the kernel launched just before it on the stream
    // (decode_prepare_kernel: ticket clear, and in the fused step the scatter / rotation of the step's rows) is
    // still running.  That kernel writes tickets, the cache rows of the step's slots and (fused step) q -- never
    // context_lens, block_tables or slot_mapping -- and everything launched before IT has completed by the time this
    // grid starts (its own blocks passed their griddepcontrol.wait before they let this grid go).  So the scan below,
    // the page lookups and the K/V rows of all other slots are settled memory: the producer requests the CTA's first
    // tiles ahead of the wait unless they hold a slot that this step writes, and waits only then.

    // The step's slots, for that check (one load latency, in parallel with the scan's).
    int my_slots[kEarlySlots];
    const bool early = p.slot_mapping == nullptr || p.B <= 32 * kEarlySlots;
    if (warp == kConsumerWarps && p.slot_mapping != nullptr && early) {
#pragma unroll
        for (int i = 0; i < kEarlySlots; ++i)
            my_slots[i] = lane + 32 * i < p.B ? __ldg(p.slot_mapping + lane + 32 * i) : -1;
    }

    // ---- prologue: total cost units per head, and where on the line every thread's share of the sequences starts ----
    // Every CTA scans context_lens itself (B / 160 values per thread and one warp scan): that is one global
    // load latency, paid in parallel by all CTAs, and cheaper than fetching the result of a serial plan.
    const int per = (p.B + kThreads - 1) / kThreads;
    {
        const int b_lo = min(p.B, tid * per), b_hi = min(p.B, b_lo + per);
        int mine = 0;
        for (int b = b_lo; b < b_hi; ++b) {
            const int tb = tiles_of(clamp_ctx(__ldg(p.context_lens + b), max_ctx));
            mine += units_of(tb, p.item_cost);
            if (tb == 0 && b % (int)gridDim.x == (int)blockIdx.x) {
                // an empty sequence attends to nothing: its rows are zeros (one CTA writes them)
                uint4* orow = reinterpret_cast<uint4*>(p.out + (size_t)b * p.H * kD);
                for (int i = 0; i < p.H * (kD * 2 / 16); ++i) orow[i] = make_uint4(0, 0, 0, 0);
            }
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) sm_i[warp] = incl;
        __syncthreads();
        long long warp_off = 0;
        for (int w = 0; w < warp; ++w) warp_off += sm_i[w];
        sm_seg[tid] = warp_off + incl - mine;
        __syncthreads();
    }
    long long total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) total += sm_i[w];
    const Cut cut = make_cut(total, p.num_groups);
    if (total == 0 || chunk >= cut.groups) {  // less work than CTAs (uniform across the CTA)
        griddep_wait();  // this grid must not be complete before the kernel in front of it is
        return;
    }

    const uint32_t stages = ring_stages(cut);

    if (warp == kConsumerWarps) {
        // =========================== producer warp ===========================
        const uint64_t pol = policy_evict_first();
        Walk walk;
        walk.x0 = cut.bound(chunk);
        walk.x1 = cut.bound(chunk + 1);
        {
            int s = -1;  // last segment that starts at or before x0
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += __popc(__ballot_sync(0xffffffffu, sm_seg[32 * w + lane] <= walk.x0));
            walk.b = s * per;
            walk.fv = sm_seg[s];
        }
        // Lane 0 walks the CTA's tiles; the other lanes help only to compare a tile with the step's slots, until the
        // wait for the kernel in front has been passed.
        Item item;
        int left = 0;             // tiles left of `item`
        int valid = 0;            // live tokens from the next tile on
        int bi = 0, off = 0;      // its page and the offset in the page
        int phys = 0, next = 0;   // that page's block and the following page's (requested one page ahead)
        const int32_t* bt = p.block_tables;
        // Metadata of the sequence after the current one is fetched one item ahead (its length and its first
        // page: every item but a CTA's first starts at tile 0), so that a sequence boundary does not put two
        // dependent global-load latencies between two tile requests.
        int pf_b = -1, pf_ctx = 0, pf_phys = 0;
        bool waited = false, ok = true;
        uint32_t it = 0, stage = 0, parity = 1;  // parity of the stage's "empty" phase: its first filling need not wait
#pragma unroll 1
        while (true) {
            int slot = -1, flags = 0;
            if (lane == 0) {
                if (left == 0 && next_item(walk, p, max_ctx, item, pf_b, pf_ctx)) {
                    left = item.n;
                    flags = kFirst;
                    valid = item.ctx - item.t0 * kTile;
                    bi = item.t0 == 0 ? 0 : item.t0 * kTile / p.block_size;
                    off = item.t0 * kTile - bi * p.block_size;
                    bt = p.block_tables + (size_t)item.b * p.MB;
                    phys = item.b == pf_b && bi == 0 ? pf_phys : __ldg(bt + bi);
                    next = bi + 1 < p.MB ? __ldg(bt + bi + 1) : 0;
                    if (walk.b < p.B) {  // the loads are issued now and first used at the next boundary
                        pf_b = walk.b;
                        pf_ctx = __ldg(p.context_lens + walk.b);
                        pf_phys = __ldg(p.block_tables + (size_t)walk.b * p.MB);
                    }
                }
                if (left > 0) {
                    slot = (phys < 0 ? 0 : (phys >= p.NB ? p.NB - 1 : phys)) * p.block_size + off;
                    if (--left == 0) flags |= item.n == item.tb ? kLast | kWhole : kLast;
                }
            }
            if (!waited) {
                const int first_slot = __shfl_sync(0xffffffffu, slot, 0);
                bool stop = !early || first_slot < 0 || it == (p.q_in_flight ? min((uint32_t)p.q_in_flight, stages) : 2 * stages);
                if (p.slot_mapping != nullptr) {
#pragma unroll
                    for (int i = 0; i < kEarlySlots; ++i) {
                        if (32 * i >= p.B) break;
                        stop |= (uint32_t)(my_slots[i] - first_slot) < (uint32_t)kTile;
                    }
                }
                if (__any_sync(0xffffffffu, stop)) {
                    griddep_wait();
                    waited = true;
                    if (lane != 0) return;
                    for (uint32_t e = 0; p.q_in_flight && e < it; ++e)
                        if (sm_meta[e].flags & kFirst) load_q(p, smem + e * kStageBytes, full_bar + e, sm_meta[e].b, kvh);
                }
            }
            if (lane == 0) {
                uint8_t* st = smem + stage * kStageBytes;
                uint64_t* bar = full_bar + stage;
                if (it >= stages && !wait_or_abort(sm_abort, empty_bar + stage, parity)) {
                    ok = false;
                    break;
                }
                if (slot < 0) {
                    sm_meta[stage].flags = kDone;
                    mbar_arrive(bar);
                    break;
                }
                sm_meta[stage].valid = valid;
                sm_meta[stage].flags = flags;
                sm_meta[stage].b = item.b;
                if ((flags & (kLast | kWhole)) == kLast) {
                    const long long first = item.fv + p.item_cost;  // unit of the sequence's tile 0
                    sm_meta[stage].part = (chunk * p.KVH + kvh) * 2 + (item.t0 == 0 ? 1 : 0);
                    sm_meta[stage].gf = item.t0 == 0 ? chunk : cut.chunk_of(first);
                    sm_meta[stage].gl = item.t0 + item.n == item.tb ? chunk : cut.chunk_of(first + item.tb - 1);
                }
                mbar_expect_tx(bar, 2 * kTileBytes + ((flags & kFirst) ? (uint32_t)p.G * kD * 2 : 0u));
                tma_load_4d_hint(st, &tm_k, bar, 0, slot, 0, kvh, pol);
                tma_load_4d_hint(st + kTileBytes, &tm_v, bar, 0, slot, 0, kvh, pol);
                if ((waited || !p.q_in_flight) && (flags & kFirst)) load_q(p, st, bar, item.b, kvh);
                valid -= kTile;
                off += kTile;
                if (off == p.block_size) {
                    off = 0;
                    phys = next;
                    ++bi;
                    next = bi + 1 < p.MB ? __ldg(bt + bi + 1) : 0;
                }
            }
            ++it;
            if (++stage == stages) stage = 0, parity ^= 1u;
        }
        if (!ok) {
            *sm_abort = 1;
            atomicOr(&g_error_flag, 1);
            // Let loads already issued land before the CTA's shared memory is released.
            for (uint32_t j = (it >= stages ? it - stages : 0); j < it; ++j)
                (void)mbar_wait(full_bar + (j % stages), (j / stages) & 1u, polls_of_ms(90));
        }
        return;
    }

    // ============================= consumer warps =============================
    // Both products are computed transposed, tokens or dims as the 16 rows and the query heads as the 8 columns of
    // mma.m16n8k16: S^T = K Q^T and O^T += V^T P^T.  Lane l holds tokens (dims) l / 4 and l / 4 + 8 of heads 2 (l % 4) and
    // 2 (l % 4) + 1.
    const int grp = lane >> 2;
    const int quad = lane & 3;
    const int mi = lane >> 3;        // which 8x8 matrix this lane addresses in ldmatrix.x4
    const int r8 = lane & 7;
    const int tok_base = warp * 16;
    const int ctid = tid;            // 0..127 among consumers
    uint32_t item = 0;
    uint32_t qb[8][2];               // Q^T: dims 16 ks + 2 quad (+1), + 8 of head grp
    float o[8][4];                   // O^T: dims 16 j + grp and + 8 of the lane's two heads
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;  // per head; the sums are this lane's tokens only
    bool waited = false;             // for the kernel in front, which clears the tickets

    for (uint32_t next = 0, parity = 0;;) {
        const uint32_t stage = next;
        if (!wait_or_abort(sm_abort, full_bar + stage, parity)) {
            *sm_abort = 1;
            atomicOr(&g_error_flag, 2);
            break;
        }
        if (++next == stages) next = 0, parity ^= 1u;
        uint8_t* st = smem + stage * kStageBytes;
        const int2 head = *reinterpret_cast<const int2*>(sm_meta + stage);
        const int flags = head.y;
        if (flags & kDone) break;
        if (flags & kFirst) {
            const uint32_t* qs = reinterpret_cast<const uint32_t*>(st + 2 * kTileBytes);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                qb[ks][0] = grp < p.G ? qs[grp * 64 + ks * 8 + quad] : 0u;
                qb[ks][1] = grp < p.G ? qs[grp * 64 + ks * 8 + 4 + quad] : 0u;
            }
            m0 = m1 = -INFINITY;
            l0 = l1 = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
        }
        const int valid = head.x - tok_base;  // live tokens in this warp's 16-token slice
        if (valid > 0) {
            const uint32_t kbase = smem_u32(st);
            const uint32_t vbase = kbase + kTileBytes;
            if (valid < 16) {
                // Rows past the context end may hold anything (even NaN bit patterns): zero the V rows so
                // that 0 * garbage cannot reach the accumulators.  Each row is 2 panels x 8 chunks of 16 B.
                for (int idx = lane; idx < (16 - valid) * 16; idx += 32) {
                    const int r = tok_base + valid + (idx >> 4);
                    const int c = idx & 15;
                    uint8_t* dst = st + kTileBytes + (c >> 3) * kPanelBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async_smem();  // order these generic writes before the stage's next TMA refill
                __syncwarp();
            }
            // ---- S^T = K Q^T for 16 tokens, in two accumulators (half the chain) ----
            float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
            {
                const uint32_t krow = kbase + (tok_base + (mi & 1) * 8 + r8) * 128;
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const int chunk = ks * 2 + (mi >> 1);
                    uint32_t a[4];
                    ldsm_x4(krow + (chunk >> 3) * kPanelBytes + (((chunk & 7) ^ r8) << 4), a);
                    mma_16816(ks & 1 ? sb : sa, a, qb[ks][0], qb[ks][1]);
                }
            }
            // ---- online softmax (log2 domain), against a maximum that may be stale by up to 2^kStale: it cancels in
            // the final division, and as long as no score exceeds it by more the lanes need not agree on a new one ----
            const float s00 = sa[0] + sb[0], s01 = sa[1] + sb[1], s10 = sa[2] + sb[2], s11 = sa[3] + sb[3];
            const bool in0 = grp < valid, in1 = grp + 8 < valid;
            float x00 = in0 ? fmaf(s00, p.scale_log2, -m0) : -INFINITY, x01 = in0 ? fmaf(s01, p.scale_log2, -m1) : -INFINITY;
            float x10 = in1 ? fmaf(s10, p.scale_log2, -m0) : -INFINITY, x11 = in1 ? fmaf(s11, p.scale_log2, -m1) : -INFINITY;
            if (__any_sync(0xffffffffu, fmaxf(fmaxf(x00, x01), fmaxf(x10, x11)) > kStale)) {
                float r0 = fmaxf(in0 ? s00 * p.scale_log2 : -INFINITY, in1 ? s10 * p.scale_log2 : -INFINITY);
                float r1 = fmaxf(in0 ? s01 * p.scale_log2 : -INFINITY, in1 ? s11 * p.scale_log2 : -INFINITY);
#pragma unroll
                for (int step = 4; step < 32; step <<= 1) {
                    r0 = fmaxf(r0, __shfl_xor_sync(0xffffffffu, r0, step));
                    r1 = fmaxf(r1, __shfl_xor_sync(0xffffffffu, r1, step));
                }
                r0 = fmaxf(m0, r0), r1 = fmaxf(m1, r1);
                const float f0 = fast_exp2(m0 - r0), f1 = fast_exp2(m1 - r1);
                m0 = r0, m1 = r1;
                l0 *= f0, l1 *= f1;
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j][0] *= f0, o[j][1] *= f1, o[j][2] *= f0, o[j][3] *= f1;
                x00 = in0 ? fmaf(s00, p.scale_log2, -m0) : -INFINITY, x01 = in0 ? fmaf(s01, p.scale_log2, -m1) : -INFINITY;
                x10 = in1 ? fmaf(s10, p.scale_log2, -m0) : -INFINITY, x11 = in1 ? fmaf(s11, p.scale_log2, -m1) : -INFINITY;
            }
            x00 = fast_exp2(x00), x01 = fast_exp2(x01), x10 = fast_exp2(x10), x11 = fast_exp2(x11);
            l0 += x00 + x10;
            l1 += x01 + x11;
            // P^T as the B operand: tokens along k, head grp as the column
            const uint32_t p0 = transpose_8x8(pack_bf16(x00, x01)), p1 = transpose_8x8(pack_bf16(x10, x11));
            // ---- O^T += V^T P^T: 8 row tiles of 16 dims ----
            {
                const uint32_t vrow = vbase + (tok_base + (mi >> 1) * 8 + r8) * 128;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int chunk = j * 2 + (mi & 1);
                    uint32_t a[4];
                    ldsm_x4_t(vrow + (chunk >> 3) * kPanelBytes + (((chunk & 7) ^ r8) << 4), a);
                    mma_16816(o[j], a, p0, p1);
                }
            }
        }
        TileMeta tm;
        if (flags & kLast) tm = sm_meta[stage];
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar + stage);
        if (!(flags & kLast)) continue;

        // ---- merge the four warps' (m, l, O) and emit the item ----
        // (m, l) exchange buffers alternate between consecutive items so that a warp that races ahead
        // into the next item cannot overwrite values a slower warp is still reading.
        float* sm_m = sm_ml + (item & 1u) * (2 * kConsumerWarps * kMaxG);
        float* sm_l = sm_m + kConsumerWarps * kMaxG;
        ++item;
#pragma unroll
        for (int step = 4; step < 32; step <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, step);
            l1 += __shfl_xor_sync(0xffffffffu, l1, step);
        }
        if (grp == 0) {
            *reinterpret_cast<float2*>(sm_m + warp * kMaxG + 2 * quad) = make_float2(m0, m1);
            *reinterpret_cast<float2*>(sm_l + warp * kMaxG + 2 * quad) = make_float2(l0, l1);
        }
        named_barrier_sync(1, kConsumerWarps * 32);
        {
            // Fixed-order reduction (bitwise reproducible): warps 0,1 store, warps 2,3 add, readers sum the two.
            float t0 = -INFINITY, t1 = -INFINITY;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) {
                const float2 v = *reinterpret_cast<const float2*>(sm_m + w * kMaxG + 2 * quad);
                t0 = fmaxf(t0, v.x), t1 = fmaxf(t1, v.y);
            }
            const float f0 = (m0 == -INFINITY) ? 0.f : fast_exp2(m0 - t0), f1 = (m1 == -INFINITY) ? 0.f : fast_exp2(m1 - t1);
            float* d0 = Os + (warp & 1) * (kMaxG * kOsStride) + 2 * quad * kOsStride + grp;
            float* d1 = d0 + kOsStride;
            if (warp < 2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    d0[16 * j] = o[j][0] * f0, d1[16 * j] = o[j][1] * f1;
                    d0[16 * j + 8] = o[j][2] * f0, d1[16 * j + 8] = o[j][3] * f1;
                }
            }
            named_barrier_sync(1, kConsumerWarps * 32);
            if (warp >= 2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    d0[16 * j] += o[j][0] * f0, d1[16 * j] += o[j][1] * f1;
                    d0[16 * j + 8] += o[j][2] * f0, d1[16 * j + 8] += o[j][3] * f1;
                }
            }
        }
        named_barrier_sync(1, kConsumerWarps * 32);
        // thread t finishes row t / 16, dims 8 (t % 16) .. + 7
        const int r = ctid >> 4, c8 = (ctid & 15) * 8;
        if (r < p.G) {
            float mt = -INFINITY;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) mt = fmaxf(mt, sm_m[w * kMaxG + r]);
            float lt = 0.f;
#pragma unroll
            for (int w = 0; w < kConsumerWarps; ++w) {
                const float mw = sm_m[w * kMaxG + r];
                if (mw != -INFINITY) lt += sm_l[w * kMaxG + r] * fast_exp2(mw - mt);
            }
            const float* s0 = Os + r * kOsStride + c8;
            const float* s1 = s0 + kMaxG * kOsStride;
            const float4 x0 = *reinterpret_cast<const float4*>(s0), x1 = *reinterpret_cast<const float4*>(s0 + 4);
            const float4 y0 = *reinterpret_cast<const float4*>(s1), y1 = *reinterpret_cast<const float4*>(s1 + 4);
            float4 a = make_float4(x0.x + y0.x, x0.y + y0.y, x0.z + y0.z, x0.w + y0.w);
            float4 b = make_float4(x1.x + y1.x, x1.y + y1.y, x1.z + y1.z, x1.w + y1.w);
            if (tm.flags & kWhole) {
                const float den = lt + 1e-9f;
                uint4 w;
                w.x = pack_bf16(a.x / den, a.y / den);
                w.y = pack_bf16(a.z / den, a.w / den);
                w.z = pack_bf16(b.x / den, b.y / den);
                w.w = pack_bf16(b.z / den, b.w / den);
                *reinterpret_cast<uint4*>(p.out + ((size_t)tm.b * p.H + (size_t)kvh * p.G + r) * kD + c8) = w;
            } else {
                float* part = p.partials + (size_t)tm.part * partial_floats(p.G);
                *reinterpret_cast<float4*>(part + r * kD + c8) = a;
                *reinterpret_cast<float4*>(part + r * kD + c8 + 4) = b;
                if (c8 == 0) {
                    part[p.G * kD + r] = mt;
                    part[p.G * kD + kMaxG + r] = lt;
                }
            }
        }
        if (!(tm.flags & kWhole)) {
            if (!waited) griddep_wait();
            waited = true;
            // Publish the partial, then take a ticket for this (sequence, kv head).  Whoever draws the last
            // ticket finds every partial of the sequence visible and combines them; nobody waits.
            named_barrier_sync(1, kConsumerWarps * 32);
            if (ctid == 0) {
                // release: the other threads' stores too, which the barrier orders before it
                sm_i[9] = (int)atomic_add_acq_rel(p.tickets + (size_t)tm.b * p.KVH + kvh, 1u);
            }
            named_barrier_sync(1, kConsumerWarps * 32);
            if (sm_i[9] == tm.gl - tm.gf) merge_sequence(p, tm.b, kvh, tm.gf, tm.gl, ctid);
        }
    }
}

// Clears the tickets of one decode call and, in the fused decode step, scatters the step's new K/V rows into
// the cache (blocks [0, store_blocks) do the scatter, the rest clear).  Runs right before paged_decode_kernel
// on the same stream.
template <typename SrcT>
__global__ void __launch_bounds__(kStoreThreads)
decode_prepare_kernel(unsigned int* __restrict__ tickets, int num_tickets, int store_blocks,
                      const SrcT* __restrict__ k, const SrcT* __restrict__ v, __nv_bfloat16* __restrict__ k_cache,
                      __nv_bfloat16* __restrict__ v_cache, const int32_t* __restrict__ slot_mapping,
                      int64_t total_chunks, int row_chunks, int64_t num_slots) {
    griddep_wait();  // the previous kernel may still be reading these tickets or the cache rows written below
    griddep_launch_dependents();
    if ((int)blockIdx.x < store_blocks) {
        store_block<SrcT, 1>(blockIdx.x, threadIdx.x, k, v, k_cache, v_cache, slot_mapping, total_chunks, row_chunks, num_slots);
    } else {
        const int i = ((int)blockIdx.x - store_blocks) * kStoreThreads + threadIdx.x;
        if (i < num_tickets) tickets[i] = 0u;
    }
}

// The same with the whole pre-attention step in front: blocks [0, pre_blocks) normalise and rotate the step's q and
// k rows and scatter the k and v rows (pre_attention.cuh), the rest clear the tickets.
// Small blocks: three of them fit an SM beside two CTAs of the attention kernel (registers).
__global__ void __launch_bounds__(preattn::kThreads)
decode_prepare_fused_kernel(unsigned int* __restrict__ tickets, int num_tickets, int pre_blocks, const preattn::Params pp) {
    griddep_wait();
    griddep_launch_dependents();
    if ((int)blockIdx.x < pre_blocks) {
        preattn::pre_attention_block(blockIdx.x, pp);
    } else {
        const int i = ((int)blockIdx.x - pre_blocks) * preattn::kThreads + threadIdx.x;
        if (i < num_tickets) tickets[i] = 0u;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int main_grid() { return kCtasPerSm * sm_count(); }

// NVLLM_B200_ITEM_COST overrides the boundary weight of the stream-K partition (an experiment knob; 0 = by tiles only).
static int item_cost() {
    static const int v = [] {
        const char* e = getenv("NVLLM_B200_ITEM_COST");
        const int x = e ? atoi(e) : kItemCostDefault;
        return x < 0 ? 0 : (x > 64 ? 64 : x);
    }();
    return v;
}

static size_t round256(size_t x) { return (x + 255) & ~size_t(255); }

static size_t ticket_bytes(int B, int KVH) { return round256((size_t)B * KVH * 4); }
static size_t partial_bytes(int ctas, int G) { return round256((size_t)ctas * 2 * partial_floats(G) * 4); }

// Tensor maps of the caches seen so far, keyed by what they encode (base address, slots, kv heads).  Encoding
// one costs the host a microsecond or two per call; a serving loop hands over the same few caches for ever.
// A map holds no reference to the memory: an entry stays valid for any later buffer with the same key.
static int cached_cache_map(CUtensorMap* map, const void* base, int64_t num_slots, int KVH) {
    struct Entry {
        const void* base;
        int64_t num_slots;
        int kvh, dev;
        CUtensorMap map;
    };
    constexpr int kEntries = 256;  // two per layer of a 128-layer model
    static std::mutex mu;
    static Entry table[kEntries];
    static int used = 0, next = 0;
    int dev = 0;
    NVLLM_CUDA_OK(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lock(mu);
        for (int i = 0; i < used; ++i) {
            const Entry& e = table[i];
            if (e.base == base && e.num_slots == num_slots && e.kvh == KVH && e.dev == dev) {
                memcpy(map, &e.map, sizeof(CUtensorMap));
                return NVLLM_B200_OK;
            }
        }
    }
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(NVLLM_B200_EDRIVER, "cuTensorMapEncodeTiled entry point not available");
    // The head dimension is seen as two halves of 64 (the widest row a 128-byte swizzle takes) with the half as an outer
    // dimension: one load then brings the tile in as the two 64-dim panels.
    cuuint64_t dims[4] = {64, (cuuint64_t)num_slots, 2, (cuuint64_t)KVH};
    cuuint64_t strides[3] = {(cuuint64_t)KVH * kD * 2, 64 * 2, (cuuint64_t)kD * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)kTile, 2, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(NVLLM_B200_EDRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    std::lock_guard<std::mutex> lock(mu);
    Entry& e = table[used < kEntries ? used++ : (next = (next + 1) % kEntries)];
    e.base = base;
    e.num_slots = num_slots;
    e.kvh = KVH;
    e.dev = dev;
    memcpy(&e.map, map, sizeof(CUtensorMap));
    return NVLLM_B200_OK;
}

static int ensure_smem_attr() {
    static std::mutex mu;
    static bool done[64];
    int dev = 0;
    NVLLM_CUDA_OK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        NVLLM_CUDA_OK(cudaFuncSetAttribute(paged_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        done[dev] = true;
    }
    return NVLLM_B200_OK;
}

// What every decode entry point shares: the argument checks and the two launches.  `tickets` / `partials` point
// into whatever scratch the entry point owns; `step` (may be null) adds the scatter of the step's new K/V rows
// to the first launch.
struct DecodeArgs {
    const void *q, *k_cache, *v_cache;
    const int32_t *block_tables, *context_lens;
    void* out;
    int B, H, KVH, D, NB, block_size, MB;
    float scale;
    void* stream;
};
struct StepArgs {
    const void *k, *v;
    const int32_t* slot_mapping;
    int src_dtype;
};

static int check_decode_args(const char* who, const DecodeArgs& a) {
    if (a.B < 0 || a.H <= 0 || a.KVH <= 0 || a.NB <= 0 || a.block_size <= 0 || a.MB <= 0)
        return fail(NVLLM_B200_EINVAL, "%s: non-positive size (B=%d H=%d KVH=%d NB=%d block=%d MB=%d)", who, a.B, a.H,
                    a.KVH, a.NB, a.block_size, a.MB);
    if (a.D != kD) return fail(NVLLM_B200_EUNSUPPORTED, "%s: head_dim %d (only 128)", who, a.D);
    if (a.block_size % kTile != 0)
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: block_size %d must be a multiple of %d", who, a.block_size, kTile);
    if (a.H % a.KVH != 0 || a.H / a.KVH > kMaxG)
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: H/KVH = %d/%d must be an integer <= %d", who, a.H, a.KVH, kMaxG);
    if ((long long)a.MB * a.block_size > 0x3fffffffLL || (long long)a.NB * a.block_size > 0x7fffffffLL)
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: cache or context too large for 32-bit token indices", who);
    if ((long long)a.B * a.KVH > 0x3fffffffLL) return fail(NVLLM_B200_EUNSUPPORTED, "%s: batch too large", who);
    return NVLLM_B200_OK;
}

static int check_decode_pointers(const char* who, const DecodeArgs& a) {
    if (!a.q || !a.k_cache || !a.v_cache || !a.block_tables || !a.context_lens || !a.out)
        return fail(NVLLM_B200_EINVAL, "%s: null pointer", who);
    if (((uintptr_t)a.q | (uintptr_t)a.k_cache | (uintptr_t)a.v_cache | (uintptr_t)a.out) & 15)
        return fail(NVLLM_B200_EINVAL, "%s: q/k_cache/v_cache/out must be 16-byte aligned", who);
    if (a.KVH > main_grid())
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: KVH %d exceeds the CTA count %d", who, a.KVH, main_grid());
    return NVLLM_B200_OK;
}

static int launch_decode(const char* who, const DecodeArgs& a, const StepArgs* step, unsigned int* tickets,
                         float* partials, const preattn::Params* pre = nullptr) {
    int rc = ensure_smem_attr();
    if (rc) return rc;
    CUtensorMap tm_k, tm_v;
    const int64_t num_slots = (int64_t)a.NB * a.block_size;
    if ((rc = cached_cache_map(&tm_k, a.k_cache, num_slots, a.KVH))) return rc;
    if ((rc = cached_cache_map(&tm_v, a.v_cache, num_slots, a.KVH))) return rc;

    Params p;
    p.q = (const __nv_bfloat16*)a.q;
    p.block_tables = a.block_tables;
    p.context_lens = a.context_lens;
    p.slot_mapping = pre ? pre->slot_mapping : (step ? step->slot_mapping : nullptr);
    p.out = (__nv_bfloat16*)a.out;
    p.tickets = tickets;
    p.partials = partials;
    p.B = a.B;
    p.H = a.H;
    p.KVH = a.KVH;
    p.G = a.H / a.KVH;
    p.NB = a.NB;
    p.block_size = a.block_size;
    p.MB = a.MB;
    p.num_groups = main_grid() / a.KVH;
    // q is requested when the tiles ahead of the wait for it have been walked.  One tile where a chunk is part of a sequence: nothing
    // can be done with more before q is here (12 sequences of 64..2000 tokens, 5 / 1 heads, 11.3 us per layer, a ring of tiles 12.0).
    // A ring where a chunk holds several: their boundaries and page lookups are then behind it (96 of 20..300, 32 / 8, 22.8 us, one
    // tile 23.4).
    p.q_in_flight = pre == nullptr ? 0 : (a.B >= p.num_groups ? kStages : 1);
    p.item_cost = item_cost();
    p.scale_log2 = a.scale * 1.4426950408889634f;

    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = reinterpret_cast<cudaStream_t>(a.stream);
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;

    const int num_tickets = a.B * a.KVH;
    const int clear_blocks = (num_tickets + kStoreThreads - 1) / kStoreThreads;
    const int row_chunks = a.KVH * kD / 8;
    const int64_t total_chunks = step ? (int64_t)a.B * row_chunks : 0;
    const int64_t store_blocks = step ? store_blocks_for(total_chunks, 1) : 0;
    if (store_blocks + clear_blocks > 0x7fffffffLL) return fail(NVLLM_B200_EUNSUPPORTED, "%s: batch too large", who);
    cfg.gridDim = dim3((unsigned)(store_blocks + clear_blocks));
    cfg.blockDim = dim3(kStoreThreads);
    cfg.dynamicSmemBytes = 0;
    if (pre) {
        const int64_t pre_blocks = preattn::blocks_for(pre->T, pre->H, pre->KVH);
        cfg.gridDim = dim3((unsigned)(pre_blocks + (num_tickets + preattn::kThreads - 1) / preattn::kThreads));
        cfg.blockDim = dim3(preattn::kThreads);
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, decode_prepare_fused_kernel, tickets, num_tickets, (int)pre_blocks, *pre));
    } else if (step && step->src_dtype == NVLLM_B200_DTYPE_F32) {
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, decode_prepare_kernel<float>, tickets, num_tickets, (int)store_blocks,
                                         (const float*)step->k, (const float*)step->v, (__nv_bfloat16*)a.k_cache,
                                         (__nv_bfloat16*)a.v_cache, step->slot_mapping, total_chunks, row_chunks,
                                         num_slots));
    } else {
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, decode_prepare_kernel<__nv_bfloat16>, tickets, num_tickets,
                                         (int)store_blocks, (const __nv_bfloat16*)(step ? step->k : nullptr),
                                         (const __nv_bfloat16*)(step ? step->v : nullptr), (__nv_bfloat16*)a.k_cache,
                                         (__nv_bfloat16*)a.v_cache, step ? step->slot_mapping : nullptr, total_chunks,
                                         row_chunks, num_slots));
    }
    cfg.gridDim = dim3((unsigned)(p.num_groups * a.KVH));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, paged_decode_kernel, tm_k, tm_v, p));
    return NVLLM_B200_OK;
}

static int decode_with_workspace(const char* who, const DecodeArgs& a, const StepArgs* step, void* workspace,
                                 size_t workspace_bytes, const preattn::Params* pre = nullptr) {
    int rc = check_decode_args(who, a);
    if (rc) return rc;
    if (step) {
        if (step->src_dtype != NVLLM_B200_DTYPE_BF16 && step->src_dtype != NVLLM_B200_DTYPE_F32)
            return fail(NVLLM_B200_EUNSUPPORTED, "%s: src_dtype %d", who, step->src_dtype);
    }
    if (a.B == 0) return NVLLM_B200_OK;
    if ((rc = check_decode_pointers(who, a))) return rc;
    if (step) {
        if (!step->k || !step->v || !step->slot_mapping) return fail(NVLLM_B200_EINVAL, "%s: null pointer", who);
        if (((uintptr_t)step->k | (uintptr_t)step->v) & 15)
            return fail(NVLLM_B200_EINVAL, "%s: k/v must be 16-byte aligned", who);
    }
    const size_t need = nvllm_b200_paged_decode_workspace_bytes(a.B, a.H, a.KVH, a.D, a.MB, a.block_size);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255))
        return fail(NVLLM_B200_EWORKSPACE, "%s: workspace of %zu bytes (256-byte aligned) required, got %zu", who, need,
                    workspace ? workspace_bytes : (size_t)0);
    return launch_decode(who, a, step, (unsigned int*)workspace,
                         (float*)((uint8_t*)workspace + ticket_bytes(a.B, a.KVH)), pre);
}

}  // namespace decode
}  // namespace nvllm

extern "C" size_t nvllm_b200_paged_decode_workspace_bytes(int B, int H, int KVH, int D, int MB, int block_size) {
    using namespace nvllm::decode;
    (void)D;
    (void)MB;
    (void)block_size;
    if (B < 0 || H <= 0 || KVH <= 0 || H % KVH != 0) return 256;
    return ticket_bytes(B, KVH) + partial_bytes(main_grid(), H / KVH) + 256;
}

extern "C" int nvllm_b200_paged_decode(const void* q, const void* k_cache, const void* v_cache,
                                       const int32_t* block_tables, const int32_t* context_lens, void* out,
                                       void* workspace, size_t workspace_bytes, int B, int H, int KVH, int D, int NB,
                                       int block_size, int MB, float scale, void* stream) {
    using namespace nvllm::decode;
    const DecodeArgs a = {q, k_cache, v_cache, block_tables, context_lens, out, B, H, KVH, D, NB, block_size, MB, scale,
                          stream};
    return decode_with_workspace("paged_decode", a, nullptr, workspace, workspace_bytes);
}

extern "C" int nvllm_b200_decode_step(const void* q, const void* k, const void* v, void* k_cache, void* v_cache,
                                      const int32_t* slot_mapping, const int32_t* block_tables,
                                      const int32_t* context_lens, void* out, void* workspace, size_t workspace_bytes,
                                      int B, int H, int KVH, int D, int NB, int block_size, int MB, float scale,
                                      int src_dtype, void* stream) {
    using namespace nvllm::decode;
    const DecodeArgs a = {q, k_cache, v_cache, block_tables, context_lens, out, B, H, KVH, D, NB, block_size, MB, scale,
                          stream};
    const StepArgs s = {k, v, slot_mapping, src_dtype};
    return decode_with_workspace("decode_step", a, &s, workspace, workspace_bytes);
}

namespace nvllm {
namespace preattn {
int check_args(const char* who, const void* q, const void* k, const void* v, const float* q_weight, const float* k_weight,
               const float* cos_sin_cache, const int32_t* positions, const void* k_cache, const void* v_cache,
               const int32_t* slot_mapping, int64_t T, int H, int KVH, int D, int64_t num_slots, int64_t max_pos);
}
}  // namespace nvllm

extern "C" int nvllm_b200_fused_decode_step(void* q, void* k, const void* v, const float* q_weight, const float* k_weight,
                                            const float* cos_sin_cache, const int32_t* positions, int64_t max_pos,
                                            float eps, void* k_cache, void* v_cache, const int32_t* slot_mapping,
                                            const int32_t* block_tables, const int32_t* context_lens, void* out,
                                            void* workspace, size_t workspace_bytes, int B, int H, int KVH, int D, int NB,
                                            int block_size, int MB, float scale, void* stream) {
    using namespace nvllm;
    using namespace nvllm::decode;
    const int64_t num_slots = (int64_t)NB * block_size;
    int rc = preattn::check_args("fused_decode_step", q, k, v, q_weight, k_weight, cos_sin_cache, positions, k_cache, v_cache,
                                 slot_mapping, B, H, KVH, D, num_slots, max_pos);
    if (rc) return rc;
    const DecodeArgs a = {q, k_cache, v_cache, block_tables, context_lens, out, B, H, KVH, D, NB, block_size, MB, scale,
                          stream};
    const preattn::Params pp{(__nv_bfloat16*)q, (__nv_bfloat16*)k, (const __nv_bfloat16*)v, q_weight, k_weight,
                             cos_sin_cache, positions, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, slot_mapping,
                             (int64_t)B, H, KVH, num_slots, max_pos, eps, 1.0f};
    return decode_with_workspace("fused_decode_step", a, nullptr, workspace, workspace_bytes, &pp);
}

namespace nvllm {
int read_decode_flags(int* out) {
    NVLLM_CUDA_OK(cudaMemcpyFromSymbol(out, decode::g_error_flag, sizeof(int)));
    return NVLLM_B200_OK;
}
int clear_decode_flags() {
    const int zero = 0;
    NVLLM_CUDA_OK(cudaMemcpyToSymbol(decode::g_error_flag, &zero, sizeof(int)));
    return NVLLM_B200_OK;
}
}  // namespace nvllm

// ---------------------------------------------------------------------------
// paged decode without a caller-provided workspace
// ---------------------------------------------------------------------------
// Some hosts of this library cannot hand it scratch memory and cannot obtain any at call time: a custom-call
// handler whose operand list is fixed by the framework, running in a process where the framework's own pool
// has already reserved nearly all of HBM (so a cudaMalloc there fails or starves the pool), or a serving
// loop that must not take the device-wide synchronisation that cudaMalloc / cudaFree imply.  For them the
// split-K scratch of the decode kernels lives in this fixed array, which every device that loads the
// library carries until the process exits.
//
// Sizes are capped so the array stays small: B * KVH <= kStaticMaxTickets and a main grid of at most
// kStaticMaxCtas CTAs (2 per SM, i.e. devices with up to 160 SMs).
namespace nvllm {
namespace decode {

constexpr int kStaticMaxBatch = 4096;
constexpr int kStaticMaxTickets = kStaticMaxBatch * 8;
constexpr int kStaticMaxCtas = 320;
constexpr size_t kStaticTicketBytes = (size_t)kStaticMaxTickets * 4;
constexpr size_t kStaticPartialBytes = (size_t)kStaticMaxCtas * 2 * ((size_t)kMaxG * kD + 2 * kMaxG) * 4;
constexpr size_t kStaticScratchBytes = kStaticTicketBytes + kStaticPartialBytes;  // about 2.8 MB

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch on the current device.  In host code the array's name is only a handle
// for the runtime, never a pointer a kernel may use, so the address is looked up once per device (with that
// device current) and cached.
static int static_scratch_address(void** out) {
    static std::mutex mu;
    static void* cached[64];
    int dev = 0;
    NVLLM_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(NVLLM_B200_EUNSUPPORTED, "paged_decode_static: device ordinal %d", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!cached[dev]) {
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr)
            return fail(NVLLM_B200_ECUDA, "paged_decode_static: cudaGetSymbolAddress failed: %s",
                        cudaGetErrorString(e));
        cached[dev] = ptr;
    }
    *out = cached[dev];
    return NVLLM_B200_OK;
}

}  // namespace decode
}  // namespace nvllm

extern "C" int nvllm_b200_paged_decode_static(const void* q, const void* k_cache, const void* v_cache,
                                              const int32_t* block_tables, const int32_t* context_lens, void* out,
                                              int B, int H, int KVH, int D, int NB, int block_size, int MB,
                                              float scale, void* stream) {
    using namespace nvllm;
    using namespace nvllm::decode;
    const char* who = "paged_decode_static";
    const DecodeArgs a = {q, k_cache, v_cache, block_tables, context_lens, out, B, H, KVH, D, NB, block_size, MB, scale,
                          stream};
    int rc = check_decode_args(who, a);
    if (rc) return rc;
    if (B > kStaticMaxBatch || (long long)B * KVH > kStaticMaxTickets)
        return fail(NVLLM_B200_EWORKSPACE,
                    "paged_decode_static: batch %d x %d kv heads exceeds the built-in scratch (max %d sequences and "
                    "%d sequence-heads); use nvllm_b200_paged_decode with a caller workspace",
                    B, KVH, kStaticMaxBatch, kStaticMaxTickets);
    if (main_grid() > kStaticMaxCtas)
        return fail(NVLLM_B200_EWORKSPACE,
                    "paged_decode_static: this device needs %d CTAs, the built-in scratch holds %d; use "
                    "nvllm_b200_paged_decode with a caller workspace",
                    main_grid(), kStaticMaxCtas);
    if (B == 0) return NVLLM_B200_OK;
    if ((rc = check_decode_pointers(who, a))) return rc;
    void* scratch = nullptr;
    if ((rc = static_scratch_address(&scratch))) return rc;
    return launch_decode(who, a, nullptr, (unsigned int*)scratch, (float*)((uint8_t*)scratch + kStaticTicketBytes));
}
