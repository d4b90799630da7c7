// varlen_prefill: causal attention over packed variable-length sequences on the
// sm_100a tensor cores (tcgen05.mma, accumulators in tensor memory).
//
// Replaces variable_length_attention_prefill (reference layers/attention.py:135-279)
// and paged_prefill_attention (layers/pallas_attention.py:557-608).  Keys and values
// are either packed like the queries ([T, KVH, 128], cu_seqlens_k == cu_seqlens_q) or
// read from the paged cache through block tables (prefix-cached prefill,
// cu_seqlens_k >= cu_seqlens_q: query i of a sequence sits at position prefix + i,
// prefix = len_k - len_q; the model runner attaches the tables on a prefix hit,
// engine/model_runner.py:311-314).
//
// Work item = two 128-row Q tiles (A and B) that share every K/V tile they read.  A row is a (token, head) pair: the item takes
// a block of consecutive tokens and all q heads of one kv head, half of the heads in each tile -- both see the same keys, run
// the same number of K/V tiles and finish together -- or, where their number is odd, all of them in both tiles, which hold
// one half of the tokens each (B may then see one K/V tile more than A); see Pack.  A tiny plan kernel turns cu_seqlens into
// the list of (sequence, token block) pairs, longest causal span first; one persistent CTA per SM
// starts on the item of its number and claims the others one by one (heavy ones first, so the CTAs finish
// together), and the kv heads go in groups whose keys and values fit the L2 (head_groups).  Tensor memory and
// barriers are set up once per CTA; the loads of the next item are already in flight
// while the current one drains.  Where the host knows that there is at most one item per SM, every CTA finds its own from
// cu_seqlens instead (ShortParams), and the step's K/V scatter runs on the SMs the items leave.  Few items with many keys are cut
// into runs of K/V tiles (SplitParams), of tile A alone where SMs would idle otherwise (lone_tiles), that a small kernel behind this
// one combines.
//
// Rows that are (token, head) pairs leave fewer of them behind the sequences' ends than rows of 128 tokens of one head, and
// tiles that span few tokens cut the products short at the diagonal: 30 prompts of 65..192 tokens, 64 / 8 heads, 64.0 -> 46.7 us,
// 16 of 128..4096, 32 / 8, 880 -> 869.
//
// Per CTA (12 warps = 3 warpgroups; the first gives registers away with setmaxnreg, the softmax
// warpgroups take them):
//   warp 0      TMA producer: Q tiles once per item, then K and V tiles [128 tokens x
//               128 dims] through one five-slot mbarrier ring filled K0 V0 K1 V1 ...
//               (cp.async.bulk.tensor, 128-byte swizzle, no multicast): K(j+2) takes the
//               slot V(j-1) leaves and V(j+2) the slot K(j) leaves, so every tile is
//               requested about two tiles before it is needed.
//   warps 1, 2  MMA issuers, one thread each for Q tile A and Q tile B: S = Q K^T
//               (operands in shared memory) and O += P V (P read from tensor memory, V
//               from shared memory, MN-major), M = N = 128, K = 16 per instruction;
//               tcgen05.commit signals the mbarriers.  K(j+1) is awaited before P.V(j) is
//               issued and all commits of the pair follow the Q.K^T(j+1) MMAs, so nothing
//               is polled between the two groups of MMAs.  Warp 1 also owns the tensor-
//               memory allocation (512 columns: S_A S_B O_A O_B).
//   warp 3      claims the CTA's items and writes their records ahead into shared memory.
//   warps 4-7   softmax of tile A, warps 8-11 of tile B: one thread per query row holds
//               its S row (128 scores) in registers, keeps the running max / sum (packed
//               f32x2 math, 3-input max), writes bf16 P back over S in two halves (each
//               releases four P.V k-steps) and rescales O only when the max grew by more
//               than 2^8 (exact: the stale max is carried into the final normalisation).
//               Tiles strictly above the diagonal are skipped; of a diagonal tile each warp
//               masks the one chunk of 32 keys that its rows' limits fall into and skips
//               the chunks behind it.  The exponentials of the two tiles take turns
//               (A(0) B(0) A(1) ...): they share the four MUFU pipes, which bound the
//               kernel, and alternating keeps one tile's MMAs, score loads and row max
//               running under the other tile's exponentials.
// Measures that only pay off together (each alone hits the next bottleneck at the same level): two
// MMA issuers, the five-slot ring, the turn-taking, and -- later -- turn-taking for the exponentials
// alone together with the poll-free MMA issue order.
// Every mbarrier wait is bounded; on timeout the CTA raises a device error flag,
// stops issuing work, and still releases its tensor memory before it exits.
#include "store_kvcache.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace nvllm {
namespace prefill {

// bit 2 (4): pipeline wait timed out; bit 4 (16): sequence too long for the plan kernel; bit 5 (32): a sequence has
// fewer keys than queries, or (packed keys) a different number -- nothing is computed for that call
__device__ int g_error_flag = 0;

constexpr int kD = 128;
constexpr int kTileQ = 128;            // rows per Q tile
constexpr int kTileKV = 128;
constexpr int kThreads = 384;            // 3 warpgroups: {TMA, MMA A, MMA B, item records} | softmax A | softmax B
constexpr int kPanelBytes = 128 * 128;  // 128 rows x 64 dims bf16, 128B-swizzled
constexpr int kTileBytes = 2 * kPanelBytes;
constexpr int kSlots = 5;                // one ring for K and V tiles, filled in the order K0 V0 K1 V1 ...
constexpr int kSmemTiles = (2 + kSlots) * kTileBytes;  // Q_A Q_B | K/V ring  (224 KB)
constexpr int kSmemBytes = kSmemTiles + 512 + 1024;  // barriers and item records, alignment slack
constexpr int kMaxLevels = 4096;       // K/V tiles per sequence the plan kernel can rank items by
constexpr uint32_t kTmemCols = 512;
constexpr float kRescaleThreshold = 8.0f;  // log2 units

constexpr int kShortBlocks = 64;       // a short launch has at most so many token blocks ...
constexpr int kShortSequences = 32;    // ... of so many sequences: a lane of a warp for each

// A (sequence, token block) pair, longest causal span first: {first query token of the sequence, its query length, first
// token of the block, sequence index} and {first key token (packed keys), key length, 0, 0}.
struct Record {
    int4 q, k;
};

// What a Q tile holds: `tokens` consecutive tokens of `heads` neighbouring q heads of one kv head, token after token, and what
// the item's second tile holds beside it.  All heads of a kv head see the same keys, so the narrower the block of tokens, the
// fewer rows lie behind a sequence's end and the more of a diagonal tile is behind every row (skipped, see key_steps).
struct Pack {
    int heads, tokens;  // of a tile
    int dq, dh;         // tile B: dq tokens further, or dh heads further
    int span;           // tokens of an item
    int per_kv;         // items per kv head and token block
};
// A kv head's G q heads in one item, half of them per tile: both tiles then see the same keys and finish together.  An odd
// number goes into both tiles, which take tokens in turn (B may see one K/V tile more).  Groups of more than eight heads are
// cut into equal parts.  `lone`: items of tile A alone, twice as many (see lone_tiles).
static Pack make_pack(int G, bool lone = false) {
    int w = std::min(G, 8);
    while (G % w) --w;
    Pack k;
    k.heads = w % 2 ? w : w / 2;
    k.tokens = kTileQ / k.heads;
    k.dq = w % 2 ? k.tokens : 0;
    k.dh = w % 2 ? 0 : k.heads;
    k.span = w % 2 ? 2 * k.tokens : k.tokens;
    k.per_kv = G / w;
    if (lone) k.dq = 1 << 28, k.dh = 0, k.span = k.tokens, k.per_kv = G / k.heads;  // no tokens behind dq: no tile B
    return k;
}

struct Params {
    const int4* items;  // record 0: {number of pairs, items claimed, head groups, 0}; then the two halves of every Record
    const int32_t* block_tables;  // [B, MB] page ids, or nullptr for packed keys/values
    int MB, block_size;
    __nv_bfloat16* out;
    int H, G;
    Pack pack;
    int per_pair;  // items per (sequence, token block)
    int wide;      // out is aligned to 32 bytes
    float scale_log2;
};

// A short launch (at most one item per SM, as far as the host knows) runs without a plan kernel and carries the step's K/V
// scatter: every CTA finds its item in the device's cu_seqlens (one load latency and a few warp votes; records laid out by the
// host and passed as arguments cost 0.4 us less, 8.5 against 8.9 us for one prompt of 87 tokens, but a captured launch then
// kept the lengths of its capture).  Should the lengths make more items than CTAs by then, a CTA takes several.
struct ShortParams : Params {
    const int32_t* cu_seqlens;
    int B;
    int item_ctas;    // CTAs that take items; the others carry the scatter
    Scatter scatter;  // chunks = 0: none
};
// Few items with many keys each (a short question behind a long cached conversation): the K/V tiles of an item are cut into
// up to `splits` contiguous runs, one per CTA, which leave partial results that prefill_combine_kernel puts together.
struct SplitParams : Params {
    float* partials;  // [CTA][Q tile][kPartialFloats]
    int splits;
    int ctas;  // the launch's
};
constexpr int kPartialFloats = kTileQ * kD + 2 * kTileQ;  // O[128][128] relative to m, then m[128] (log2 units) and l[128]
// K/V tiles per run.  A row that sees none of a run's keys would have no maximum.  An item's first token sees all of its tiles
// but one (two where the item has more tokens than a tile keys).
__host__ __device__ __forceinline__ int min_run(int span) { return span > kTileKV ? 3 : 2; }
// Items of fewer tiles stay whole: they take less time than the partial results and the combining launch (about 6 us).  The
// rule looks at an item's own tiles, so that packed keys and keys in pages give the same bits.  20 new tokens behind 1200 cached
// ones, 16 / 2 heads: whole 27.6 us, cut 19.6; 100 behind 8000, 32 / 8: 130 and 35.
constexpr int kSplitTiles = 8;
constexpr int kMaxSplits = 16;  // runs per item
// A sequence without a cached prefix is cut only if it has more keys: below, whole items leave the launch short (no plan kernel, the
// scatter in it).  One prompt of 1200, 8 / 2 heads, whole 25.2 us, cut 27.5; of 1500, 8 / 1, whole 34.6, cut 28.0.
constexpr int kWholeKeys = 11 * kTileKV;
// The launch has a CTA for every run that the host could foresee.  Where the device's lengths make more items than that (a
// captured launch whose lengths were rewritten), the items stay whole and the CTAs claim them one by one.
__device__ __forceinline__ int splits_of(const SplitParams& p, int pairs) {
    return (long long)pairs * p.per_pair * p.splits <= p.ctas ? p.splits : 1;
}
__device__ __forceinline__ int runs_of(const Params& p, int splits, int n_a, int prefix, int len_k) {
    return n_a < kSplitTiles || (prefix == 0 && len_k <= kWholeKeys) ? 1 : min(splits, n_a / min_run(p.pack.span));
}

__device__ __forceinline__ Record record_of(const Params& p, int pair) {
    return Record{__ldg(p.items + 1 + 2 * pair), __ldg(p.items + 2 + 2 * pair)};
}
__device__ __forceinline__ int claim_item(const Params& p) {
    return (int)gridDim.x + atomicAdd(&const_cast<int4*>(p.items)->y, 1);
}
// The item list's header, read once per thread.
struct List {
    int pairs, groups;
};
__device__ __forceinline__ List list_of(const Params& p) {
    const int4 h = p.items[0];
    return List{h.x, h.z};
}
__device__ __forceinline__ int items_of(const Params& p, const List& l) { return l.pairs * p.per_pair; }
__device__ __forceinline__ int items_of(const SplitParams& p, const List& l) {
    return l.pairs * p.per_pair * splits_of(p, l.pairs);
}

// ------------------------------------------------------------------------------------------
// tcgen05 wrappers
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc)
        : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets lane (base + i), columns c..c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,"
        "%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// 32 lanes x 16 columns, from the first 16 words of r.
template <int N>
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[N]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
            taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// Packed fp32 pairs (one instruction, two lanes of math) and the three-input max of sm_100.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (sm_100).
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version
    d |= (uint64_t)2 << 61;  // SWIZZLE_128B
    return d;
}
// K-major operand tile [128 rows][128 dims] stored as two 64-dim panels; k-step = 16 dims.
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t tile_addr, int ks) {
    return make_desc(tile_addr + (ks >> 2) * kPanelBytes + (ks & 3) * 32, 16, 1024);
}
// MN-major operand: V tile [128 tokens][128 dims] as two 64-dim panels; N = dims, K = tokens; k-step = 16 tokens.
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t tile_addr, int ks) {
    return make_desc(tile_addr + ks * 16 * 128, kPanelBytes, 1024);
}

constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);
constexpr uint32_t idesc_qk(uint32_t keys) { return kIdesc | ((keys >> 3) << 17); }
constexpr uint32_t kIdescPV = kIdesc | ((128u >> 3) << 17) | (1u << 16);  // B operand MN-major

// ------------------------------------------------------------------------------------------
// plan kernel: (sequence, token block) pairs sorted by causal span, largest first
// ------------------------------------------------------------------------------------------
// Longest spans first means that all sequences are in flight at once.  Where their keys and values do not fit the L2 the kv
// heads are taken in groups whose keys and values do, one group after the other, as long as each is long enough for its CTAs to
// end together.  16 prompts of 128..4096 tokens, 32 / 8 heads (139 MB of K and V): 912 us as one group, 880 in two, 916 in eight (four
// rounds of items each); 12 of 17..700 behind 500..5000 cached ones (four rounds in all): 258, in two 271.
constexpr long long kGroupRows = (96 << 20) / 512;  // (token, kv head) rows of K and V: 512 bytes
constexpr int kGroupRounds = 6;                     // items per CTA and group
__device__ int head_groups(long long keys, int pairs, int per_pair, int KVH, int ctas) {
    int n = 1;
    while (KVH % (2 * n) == 0 && keys * KVH > kGroupRows * n &&
           (long long)pairs * per_pair >= (long long)2 * n * kGroupRounds * ctas)
        n *= 2;
    return n;
}

// K/V tiles in front of the last one that block l of a sequence sees.
__device__ __forceinline__ int level_of(int len, int len_k, int l, int span) {
    const int last = min(len, (l + 1) * span) - 1 + max(len_k - len, 0);  // position of the block's last token
    return min(last / kTileKV, kMaxLevels - 1);
}

constexpr int kPlanThreads = 1024;
__global__ void __launch_bounds__(kPlanThreads) prefill_plan_kernel(const int32_t* __restrict__ cu_seqlens,
                                                                    const int32_t* __restrict__ cu_k, int paged, int B,
                                                                    int4* __restrict__ items, int capacity, int span,
                                                                    int per_pair, int KVH, int ctas, int behind_store) {
    // A token block's level is the number of K/V tiles in front of its last one (level_of).
    __shared__ int hist[kMaxLevels];
    __shared__ int base[kMaxLevels];
    __shared__ int lengths[2][kPlanThreads];  // cu_seqlens and cu_k, where they fit and a warp takes several sequences: read at once
    __shared__ unsigned int warp_keys[kPlanThreads / 32];
    __shared__ int max_level, bad;
    // Behind this step's own scatter there is nothing to wait for: that kernel has let this one go after everything in front
    // of it was complete, and writes nothing that is read here.  The wait at the end makes the main kernel's wait cover it.
    // Only then may the main kernel start: its CTAs dealt to SMs in the order in which the scatter left them, instead of in
    // order, cost long launches 1 to 3 % (neighbouring CTAs read the same K/V tiles).
    if (!behind_store) {
        griddep_wait();
        griddep_launch_dependents();
    }
    for (int i = threadIdx.x; i < kMaxLevels; i += blockDim.x) hist[i] = 0;
    if (threadIdx.x == 0) max_level = 0, bad = 0;
    const int *q_at = cu_seqlens, *k_at = cu_k;
    if (B > kPlanThreads / 32 && B < kPlanThreads) {
        if ((int)threadIdx.x <= B) {
            lengths[0][threadIdx.x] = cu_seqlens[threadIdx.x];
            lengths[1][threadIdx.x] = cu_k[threadIdx.x];
        }
        q_at = lengths[0], k_at = lengths[1];
    }
    __syncthreads();
    // few sequences: a warp each, its lanes take the token blocks; many: a thread each
    const bool by_warp = B <= 256;
    const int b0 = by_warp ? threadIdx.x >> 5 : threadIdx.x, db = by_warp ? kPlanThreads / 32 : kPlanThreads;
    const int l0 = by_warp ? threadIdx.x & 31 : 0, dl = by_warp ? 32 : 1;
    int my_level = 0;
    unsigned int my_keys = 0;  // at most 64 sequences of 2^19 keys
    for (int b = b0; b < B; b += db) {
        const int len = q_at[b + 1] - q_at[b];
        const int len_k = k_at[b + 1] - k_at[b];
        // keys can never be fewer than queries; packed keys sit beside the queries, so the counts must be equal
        if (len > 0 && (len_k < len || (!paged && (len_k != len || k_at[b] != q_at[b])))) bad = 1;
        const int n = len > 0 ? (len - 1) / span + 1 : 0;
        if (n > 0 && l0 == 0) {
            const int tiles = (max(len, len_k) - 1) / kTileKV + 1;
            my_level = max(my_level, min(tiles, kMaxLevels));
            my_keys += (unsigned int)min(len_k, kMaxLevels * kTileKV);
            if (tiles > kMaxLevels) atomicOr(&g_error_flag, 16);
        }
        for (int l = l0; l < n; l += dl) atomicAdd(&hist[level_of(len, len_k, l, span)], 1);
    }
    // One update per warp (a 64-bit atomic of shared memory and a load latency per sequence cost 100 sequences of 10..100 tokens
    // 2.1 us of 43.3).
    my_level = __reduce_max_sync(0xffffffffu, my_level);
    my_keys = __reduce_add_sync(0xffffffffu, my_keys);
    if ((threadIdx.x & 31) == 0) {
        warp_keys[threadIdx.x >> 5] = my_keys;
        if (my_level > 0) atomicMax(&max_level, my_level);
    }
    __syncthreads();
    if (bad) {  // uniform: publish an empty list so that the main kernel computes nothing
        if (threadIdx.x == 0) {
            items[0] = make_int4(0, 0, 1, 0);
            atomicOr(&g_error_flag, 32);
        }
        if (behind_store) griddep_wait();
        return;
    }
    if (threadIdx.x < 32) {  // base[l] = number of pairs of higher levels: a warp scan from the top, 32 levels at a time
        int run = 0;
        for (int top = max_level - 1; top >= 0; top -= 32) {
            const int l = top - (int)threadIdx.x;
            const int h = l >= 0 ? hist[l] : 0;
            int incl = h;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += v;
            }
            if (l >= 0) base[l] = run + incl - h;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        const unsigned int mine = warp_keys[threadIdx.x];
        const long long keys = (long long)__reduce_add_sync(0xffffffffu, mine >> 16) * 65536 +
                               __reduce_add_sync(0xffffffffu, mine & 0xffffu);
        if (threadIdx.x == 0)
            items[0] = make_int4(min(run, capacity), 0, head_groups(keys, min(run, capacity), per_pair, KVH, ctas), 0);
    }
    __syncthreads();
    for (int b = b0; b < B; b += db) {
        const int start = q_at[b];
        const int len = q_at[b + 1] - start;
        const int len_k = k_at[b + 1] - k_at[b];
        const int n = len > 0 ? (len - 1) / span + 1 : 0;
        for (int l = l0; l < n; l += dl) {
            const int slot = atomicAdd(&base[level_of(len, len_k, l, span)], 1);
            if (slot < capacity) {
                items[1 + 2 * slot] = make_int4(start, len, l * span, b);
                items[2 + 2 * slot] = make_int4(k_at[b], len_k, 0, 0);
            }
        }
    }
    if (behind_store) {
        griddep_wait();
        griddep_launch_dependents();
    }
}

// ------------------------------------------------------------------------------------------
// main kernel
// ------------------------------------------------------------------------------------------
struct Item {
    int seq_start, len, q0, head;      // first query token of the sequence, query length, first token of the block, first head
    int k_start, len_k, prefix, kvh;   // first key token (packed keys), key length, len_k - len, kv head
    int n_a, n_b, n_kv, b;             // KV tiles seen by Q tile A, by Q tile B (0: no such rows; else n_a or n_a + 1), the
                                       // larger (0: nothing to do; -1: no more items), sequence
    int kv0;                           // a run of a split item: its first KV tile (len_k and prefix count from there on), else -1
};
constexpr int kItemRing = 2;
constexpr int kItemReaders = 3 + 8;    // TMA producer, two MMA issuers, eight softmax warps

struct Shared {
    Item items[kItemRing];  // the items of this CTA, written ahead by warp 3
    uint64_t item_full[kItemRing], item_empty[kItemRing];
    uint64_t q_full, q_empty;
    uint64_t kv_full[kSlots], kv_empty[kSlots];
    uint64_t s_full[2], p_full[2][2], o_full[2], o_empty[2];
    uint64_t turn[2];  // softmax ping-pong: turn[0] = "tile A finished a softmax", turn[1] = "tile B finished one"
    uint32_t tmem_base;
    volatile int abort_flag;
};

static_assert(sizeof(Shared) <= 512, "see kSmemBytes");

__device__ __forceinline__ bool wait_or_abort(Shared* sh, uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    if (sh->abort_flag) return false;
    if (mbar_wait(bar, parity)) return true;
    sh->abort_flag = 1;
    atomicOr(&g_error_flag, 4);
    return false;
}

// Keys up to the last one that a row of Q tile x sees, counted from the item's first K/V tile.
__device__ __forceinline__ int visible_keys(const Params& p, const Item& it, int x) {
    return it.prefix + min(it.len, it.q0 + x * p.pack.dq + p.pack.tokens);
}
// Steps of 16 keys of the tile's n-th and last K/V tile that hold any of them: what its two products go through.
__device__ __forceinline__ int key_steps(int keys, int n) { return (min(kTileKV, keys - (n - 1) * kTileKV) + 15) >> 4; }

// Item r (of per_pair) of a (sequence, token block).
__device__ __forceinline__ Item make_item(const Params& p, const Record& rec, int r) {
    Item it;
    it.kvh = r / p.pack.per_kv;
    it.head = it.kvh * p.G + (r - it.kvh * p.pack.per_kv) * (p.G / p.pack.per_kv);
    const int4 q = rec.q, k = rec.k;
    it.seq_start = q.x;
    it.len = q.y;
    it.q0 = q.z;
    it.b = q.w;
    it.k_start = k.x;
    it.len_k = k.y;
    it.prefix = it.len_k - it.len;  // >= 0: the plan kernel publishes no items otherwise
    it.n_a = (visible_keys(p, it, 0) - 1) / kTileKV + 1;
    it.n_b = it.len - it.q0 > p.pack.dq ? (visible_keys(p, it, 1) - 1) / kTileKV + 1 : 0;
    it.n_kv = max(it.n_a, it.n_b);
    it.kv0 = -1;
    return it;
}
// Items go by head group (see head_groups), in a group by pair.
__device__ __forceinline__ Item load_item(const Params& p, const List& l, int idx) {
    int per = p.per_pair, first = 0;
    if (l.groups > 1) {
        per /= l.groups;
        first = idx / (l.pairs * per) * per;
        idx -= first * l.pairs;
    }
    const int pair = idx / per;
    return make_item(p, record_of(p, pair), first + idx - pair * per);
}
__device__ __forceinline__ Item load_item(const SplitParams& p, const List& l, int idx) {
    const int splits = splits_of(p, l.pairs), c = idx % splits;
    Item it = load_item(static_cast<const Params&>(p), l, idx / splits);
    const int runs = runs_of(p, splits, it.n_a, it.prefix, it.len_k);
    if (runs == 1) {
        if (c > 0) it.n_a = it.n_b = it.n_kv = 0;
        return it;
    }
    if (c >= runs) {
        it.n_a = it.n_b = it.n_kv = 0;
        return it;
    }
    const int j0 = it.n_a * c / runs, j1 = c + 1 == runs ? it.n_kv : it.n_a * (c + 1) / runs;
    it.kv0 = j0;
    it.n_a = min(it.n_a, j1) - j0;
    it.n_b = it.n_b > 0 ? min(it.n_b, j1) - j0 : 0;
    it.n_kv = j1 - j0;
    it.len_k -= j0 * kTileKV;
    it.prefix -= j0 * kTileKV;
    return it;
}

// The next item from the ring (k-th of this CTA).  The readers arrive on the slot once they have their copy, the softmax
// warps once they are done with the item.
__device__ __forceinline__ bool next_item(Shared* sh, uint32_t k, Item& it) {
    const uint32_t slot = k % kItemRing;
    if (!wait_or_abort(sh, &sh->item_full[slot], (k / kItemRing) & 1u)) return false;
    it = sh->items[slot];
    return it.n_kv >= 0;
}

// First token (row of the k / v tensor map) of KV tile j of the item's sequence.
__device__ __forceinline__ int kv_tile_token(const Params& p, const Item& it, int j) {
    const int off = (max(it.kv0, 0) + j) * kTileKV;
    if (p.block_tables == nullptr) return it.k_start + off;
    int page = __ldg(p.block_tables + (size_t)it.b * p.MB + off / p.block_size);
    if (page < 0) page = 0;  // a padding entry: never reached for keys below len_k
    return page * p.block_size + off % p.block_size;  // block_size is a multiple of the tile: a tile never straddles pages
}

// The output is marked as evicted first, so that it does not push keys and values out of the L2 (16 prompts of 128..4096 tokens, 32 / 8
// heads, with Q's loads marked too: 931 -> 912 us as one head group).  The GEMM that reads it next does not notice: attention and an
// o_proj-shaped GEMM together, outputs of 4 to 268 MB, take 0 to 0.4 % less with the mark.
__device__ __forceinline__ void store_32bytes(void* dst, const uint32_t (&w)[8]) {
    asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// One 128-column S row -> running max, optional O rescale, bf16 P in two halves.  DIAG: key column c of this tile is
// visible iff c <= lim (lim may be negative -- nothing visible in this tile -- or >= 127), and the limits of the warp's rows
// lie in warp_lo .. warp_hi; columns behind every limit may hold anything.  alive: the warp's rows in front of the
// sequence's end; the others (the next sequence's queries, rows that no load fills) have no vote on when to rescale, or the
// live rows' bits would depend on them.  turn_bar (or null): the other tile's hand-over this tile's exponentials wait for;
// turn_out (or null): where this tile hands over.
// The whole row is held in registers (the softmax warpgroups raise their register budget with setmaxnreg), so
// tensor memory is read once and its latency is paid once per tile.
template <bool DIAG>
__device__ __forceinline__ bool softmax_tile(Shared* sh, const int x, const uint32_t t_s, const uint32_t t_o,
                                             const int lim, const int warp_lo, const int warp_hi, const bool first,
                                             const uint32_t o_parity_prev,
                                             const float scale_log2, const uint32_t alive, float& m_run, float& m_used, float& l,
                                             uint64_t* turn_bar, const uint32_t turn_parity, uint64_t* turn_out) {
    uint32_t v[4][32];
    tmem_ld32(t_s, v[0]);
    tmem_ld32(t_s + 32, v[1]);
    tmem_ld32(t_s + 64, v[2]);
    tmem_ld32(t_s + 96, v[3]);
    tmem_wait_ld();
    float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (DIAG) {
            if (32 * c > warp_hi) continue;  // nothing of this chunk is visible to any row of the warp
            if (32 * c + 31 > warp_lo) {     // mask in place so that the second pass needs no select
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (c * 32 + i > lim) v[c][i] = 0xFF800000u;
            }
        }
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            mx0 = max3(mx0, __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
            mx1 = max3(mx1, __uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
            mx2 = max3(mx2, __uint_as_float(v[c][i + 4]), __uint_as_float(v[c][i + 5]));
            mx3 = max3(mx3, __uint_as_float(v[c][i + 6]), __uint_as_float(v[c][i + 7]));
        }
    }
    m_run = fmaxf(m_run, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
    if (turn_bar != nullptr && !wait_or_abort(sh, turn_bar, turn_parity)) return false;
    if (first) {
        m_used = m_run;  // finite for live rows: key 0 of the sequence is visible to every row and sits in the first tile
    } else {
        const bool grow = (m_run - m_used) * scale_log2 > kRescaleThreshold;
        if (__ballot_sync(0xffffffffu, grow) & alive) {
            // O holds sums relative to m_used: bring it to m_run before this tile's P.V is added.
            if (!wait_or_abort(sh, &sh->o_full[x], o_parity_prev)) return false;
            tc_fence_after();
            const float f = fast_exp2((m_used - m_run) * scale_log2);
#pragma unroll 1
            for (int c = 0; c < 8; ++c) {
                uint32_t ov[16];
                tmem_ld16(t_o + c * 16, ov);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * f);
                tmem_st16(t_o + c * 16, ov);
            }
            tmem_wait_st();
            l *= f;
            m_used = m_run;
        }
    }
    // p = 2^(s*scale - m) as bf16 pairs, written over the S columns (all of them are in registers by now):
    // chunk c (scores 32c..32c+31) becomes packed columns 16c..16c+15.
    const float neg = -m_used * scale_log2;
    const uint64_t scale2 = pack2(scale_log2, scale_log2), neg2 = pack2(neg, neg);
    uint64_t acc_a = pack2(0.f, 0.f), acc_b = pack2(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (DIAG && 32 * c > warp_hi) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[c][i] = 0u;
        } else {
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            float x0, x1, x2, x3;
            unpack2(fma2(pack2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), scale2, neg2), x0, x1);
            unpack2(fma2(pack2(__uint_as_float(v[c][2 * i + 2]), __uint_as_float(v[c][2 * i + 3])), scale2, neg2), x2,
                    x3);
            const float e0 = fast_exp2(x0), e1 = fast_exp2(x1);  // 2^-inf = 0 for masked keys
            const float e2 = fast_exp2(x2), e3 = fast_exp2(x3);
            acc_a = add2(acc_a, pack2(e0, e1));
            acc_b = add2(acc_b, pack2(e2, e3));
            v[c][i] = pack_bf16(e0, e1);  // in place: word i <= 2i has been consumed
            v[c][i + 1] = pack_bf16(e2, e3);
        }
        }
        tmem_st16(t_s + c * 16, v[c]);
        if (c == 3 && turn_out != nullptr) {
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbar_arrive(turn_out);
        }
        if (c & 1) {  // a half of P (64 keys) is complete: release its four P.V k-steps
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbar_arrive(&sh->p_full[x][c >> 1]);
        }
    }
    float s0, s1, s2, s3;
    unpack2(acc_a, s0, s1);
    unpack2(acc_b, s2, s3);
    l += (s0 + s1) + (s2 + s3);
    return true;
}

template <class P>
__global__ void __launch_bounds__(kThreads, 1)
varlen_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ P p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;                                   // [2][tile]
    uint8_t* sKV = smem + 2 * kTileBytes;                 // [kSlots][tile]: ring position 2j holds K(j), 2j+1 holds V(j)
    Shared* sh = reinterpret_cast<Shared*>(smem + kSmemTiles);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    constexpr bool kShort = std::is_same<P, ShortParams>::value;
    if constexpr (kShort) {
        if ((int)blockIdx.x >= p.item_ctas) {  // a CTA that only scatters
            griddep_wait();
            const Scatter& sc = p.scatter;
            const int first = (blockIdx.x - p.item_ctas) * (kThreads / kStoreThreads) + tid / kStoreThreads;
            if (tid < kThreads / kStoreThreads * kStoreThreads)
                store_block<__nv_bfloat16>(first, tid % kStoreThreads, sc.k, sc.v, sc.k_cache, sc.v_cache, sc.slot_mapping,
                                           sc.chunks, sc.row_chunks, sc.num_slots);
            return;
        }
    }
    if (tid == 0) {
        for (int s = 0; s < kItemRing; ++s) {
            mbar_init(&sh->item_full[s], 1);
            mbar_init(&sh->item_empty[s], kItemReaders);
        }
        mbar_init(&sh->q_full, 1);
        mbar_init(&sh->q_empty, 2);   // both MMA issuers
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(&sh->kv_full[s], 1);
            mbar_init(&sh->kv_empty[s], 2);  // both MMA issuers
        }
        for (int x = 0; x < 2; ++x) {
            mbar_init(&sh->s_full[x], 1);
            mbar_init(&sh->p_full[x][0], kTileQ / 32);  // one arrival per softmax warp
            mbar_init(&sh->p_full[x][1], kTileQ / 32);
            mbar_init(&sh->o_full[x], 1);
            mbar_init(&sh->o_empty[x], kTileQ / 32);
            mbar_init(&sh->turn[x], kTileQ / 32);
        }
        sh->abort_flag = 0;
        sh->tmem_base = 0xFFFFFFFFu;
        fence_mbar_init();
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(&tm_k);
        prefetch_tensormap(&tm_v);
    }
    __syncthreads();
    if (warp == 1) {
        tmem_alloc(&sh->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;

    griddep_wait();  // the plan kernel's item list (and the caller's q/k/v) must be visible from here on

    // Register budget: the TMA / MMA warpgroup keeps 96 registers per thread, the two softmax warpgroups take 200
    // (96*128 + 200*256 <= 64K), enough to hold a whole 128-column score row.
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    if (warp == 0) {
        // =============================== TMA producer ===============================
        if (lane == 0) {
            const uint64_t once = policy_evict_first();
            uint32_t kt = 0, i = 0;
            bool ok = true;
            Item it;
            while (ok && next_item(sh, i, it)) {
                mbar_arrive(&sh->item_empty[i % kItemRing]);
                const int kvh = it.kvh;
                const int tok_q = it.seq_start + it.q0;
                if (i > 0 && !(ok = wait_or_abort(sh, &sh->q_empty, (i - 1) & 1u))) break;
                mbar_expect_tx(&sh->q_full, (it.n_b > 0 ? 4u : 2u) * 128u * (uint32_t)(p.pack.heads * p.pack.tokens));
                tma_load_3d_hint(sQ, &tm_q, &sh->q_full, 0, it.head, tok_q, once);
                tma_load_3d_hint(sQ + kPanelBytes, &tm_q, &sh->q_full, 64, it.head, tok_q, once);
                if (it.n_b > 0) {
                    tma_load_3d_hint(sQ + kTileBytes, &tm_q, &sh->q_full, 0, it.head + p.pack.dh, tok_q + p.pack.dq, once);
                    tma_load_3d_hint(sQ + kTileBytes + kPanelBytes, &tm_q, &sh->q_full, 64, it.head + p.pack.dh, tok_q + p.pack.dq, once);
                }
                for (int j = 0; j < it.n_kv; ++j, ++kt) {
                    const int tok = kv_tile_token(p, it, j);
#pragma unroll
                    for (int kv = 0; kv < 2; ++kv) {  // K(j) then V(j): with five slots both are requested ~2 tiles ahead
                        const uint32_t pos = 2 * kt + kv;
                        const int slot = pos % kSlots;
                        if (!(ok = wait_or_abort(sh, &sh->kv_empty[slot], ((pos / kSlots) & 1u) ^ 1u))) break;
                        const CUtensorMap* tm = kv == 0 ? &tm_k : &tm_v;
                        mbar_expect_tx(&sh->kv_full[slot], kTileBytes);
                        tma_load_3d(sKV + slot * kTileBytes, tm, &sh->kv_full[slot], 0, kvh, tok);
                        tma_load_3d(sKV + slot * kTileBytes + kPanelBytes, tm, &sh->kv_full[slot], 64, kvh, tok);
                    }
                    if (!ok) break;
                }
                ++i;
            }
        }
    } else if (warp == 3) {
        // ============================== item records ================================
        // The readers would each spend two dependent loads and a division per item between two items.  The first item of a
        // CTA is fixed, the others are claimed from a counter when the softmax warps start on the item before: with the
        // heaviest items first the CTAs finish together (dealt round-robin, the CTAs with the heaviest items of every round
        // also got the ones left over: 257 us for the last of 148, 209 for the median one).
        if constexpr (kShort) {
            // Lane b has sequence b.  Items go by token block, the last ones (the longest spans) first.
            const int start = lane < p.B ? __ldg(p.cu_seqlens + lane) : 0;
            const int len = lane < p.B ? __ldg(p.cu_seqlens + lane + 1) - start : 0;
            const int blocks = len > 0 ? (len - 1) / p.pack.span + 1 : 0;
            const int items = tmem != 0xFFFFFFFFu ? __reduce_add_sync(0xffffffffu, blocks) * p.per_pair : 0;
            const int levels = __reduce_max_sync(0xffffffffu, blocks);
            uint32_t k = 0;
            for (int idx = blockIdx.x, more = 1; more; idx += p.item_ctas) {
                int at = idx / p.per_pair, level = levels - 1;
                const int r = idx - at * p.per_pair;
                int4 q = make_int4(0, 0, 0, 0);
                if (idx < items) {
                    uint32_t has = __ballot_sync(0xffffffffu, blocks > level);
                    for (; at >= __popc(has); has = __ballot_sync(0xffffffffu, blocks > level)) at -= __popc(has), --level;
                    const bool mine = blocks > level && __popc(has & ((1u << lane) - 1)) == at;
                    const int b = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
                    q = make_int4(__shfl_sync(0xffffffffu, start, b), __shfl_sync(0xffffffffu, len, b), level * p.pack.span, b);
                }
                if (lane == 0) {
                    Item it;
                    it.n_kv = -1;
                    if (idx < items) it = make_item(p, Record{q, make_int4(q.x, q.y, 0, 0)}, r);
                    if (it.n_kv != 0) {
                        const uint32_t slot = k % kItemRing;
                        more = wait_or_abort(sh, &sh->item_empty[slot], ((k / kItemRing) & 1u) ^ 1u);
                        if (more) {
                            sh->items[slot] = it;
                            mbar_arrive(&sh->item_full[slot]);
                            ++k;
                            more = it.n_kv > 0;
                        }
                    }
                }
                more = __shfl_sync(0xffffffffu, more, 0);
            }
        } else if (lane == 0) {
            const List list = list_of(p);
            const int total = tmem != 0xFFFFFFFFu ? items_of(p, list) : 0;
            uint32_t k = 0;
            int idx = blockIdx.x;
            while (true) {
                const uint32_t slot = k % kItemRing;
                if (!wait_or_abort(sh, &sh->item_empty[slot], ((k / kItemRing) & 1u) ^ 1u)) break;
                Item it;
                do {
                    if (k > 0 || idx != (int)blockIdx.x) idx = claim_item(p);
                    it.n_kv = -1;
                    if (idx < total) it = load_item(p, list, idx);
                    if (it.n_kv == 0) idx = total;  // nothing to do there: claim another one
                } while (it.n_kv == 0);
                sh->items[slot] = it;
                mbar_arrive(&sh->item_full[slot]);
                if (it.n_kv < 0) break;
                ++k;
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ============================== MMA issuers ===============================
        // One issuing thread per Q tile (warp 1: tile A, warp 2: tile B).  An issuing thread blocks on every
        // tcgen05.mma until the tensor pipe accepts it and pays a couple of hundred cycles for every barrier it
        // polls; with two independent issuers one tile's bookkeeping hides behind the other tile's MMAs.  Each
        // thread owns its tile's S / P / O barriers; the shared K/V ring slots and the Q buffer are released by
        // both (their "empty" barriers count two arrivals: a tcgen05.commit from a thread that read the slot, a
        // plain arrive from a thread whose tile does not need it).
        if (lane == 0) {
            const int x = warp - 1;
            const uint32_t s_t = tmem + x * 128, o_t = tmem + 256 + x * 128;
            // Descriptors are built once: per k-step and per ring slot only the 14-bit start-address field
            // (bytes >> 4) moves, so issuing an MMA costs one 32-bit add instead of a descriptor rebuild.
            const uint64_t q_desc = kmajor_desc(smem_u32(sQ + x * kTileBytes), 0);
            const uint64_t k_desc0 = kmajor_desc(smem_u32(sKV), 0), v_desc0 = mnmajor_desc(smem_u32(sKV), 0);
            constexpr uint32_t kSlotStep = (uint32_t)(kTileBytes >> 4);  // next ring slot, in descriptor address units
            uint32_t kt = 0;     // K/V tiles consumed before this item
            uint32_t tiles = 0;  // tiles finished by this Q tile, over all items (barrier phases)
            uint32_t used = 0;   // items in which this Q tile was active (o_empty phases)
            uint32_t i = 0;      // items
            bool ok = true;

            // behind_pv: o_full(j-1) is committed in front of s_full(j), so that a softmax warp that has seen S(j) finds that
            // phase of o_full complete.  The other way round a warp that skips the softmax (its rows lie behind the
            // sequence's end) could be at its wait for o_full(j) a phase too early, where the parity aliases.
            //
            // A tile's last products leave out the keys behind every row (key_steps).  They are code of their own: with the key
            // count as a variable in the others long prompts were 2 % slower (1 of 8192 tokens, 64 / 8 heads: 1049 -> 1074 us).
            auto issue_qk = [&](uint64_t kd, bool behind_pv, auto last, int steps) {
                if constexpr (decltype(last)::value) {
                    const uint32_t idesc = idesc_qk(16 * steps);
#pragma unroll 1
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t step = (uint32_t)(((ks >> 2) * kPanelBytes + (ks & 3) * 32) >> 4);
                        mma_ss(s_t, q_desc + step, kd + step, idesc, ks > 0);
                    }
                } else {
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        const uint32_t step = (uint32_t)(((ks >> 2) * kPanelBytes + (ks & 3) * 32) >> 4);
                        mma_ss(s_t, q_desc + step, kd + step, idesc_qk(kTileKV), ks > 0);
                    }
                }
                if (behind_pv) tc_commit(&sh->o_full[x]);
                tc_commit(&sh->s_full[x]);
            };
            auto issue_pv = [&](int j, uint64_t vd, auto last, int steps) -> bool {
                if (j == 0 && used > 0 && !wait_or_abort(sh, &sh->o_empty[x], (used - 1) & 1u)) return false;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (!wait_or_abort(sh, &sh->p_full[x][half], tiles & 1u)) return false;
                    tc_fence_after();
#pragma unroll
                    for (int ks = half * 4; ks < half * 4 + 4; ++ks)
                        if (!decltype(last)::value || ks < steps)
                            mma_ts(o_t, s_t + ks * 8, vd + (uint32_t)((ks * 16 * 128) >> 4), kIdescPV, (j > 0 || ks > 0));
                }
                ++tiles;
                return true;
            };
            // the slot holding ring position pos: K(j) sits at 2j, V(j) at 2j+1
            auto slot_full = [&](uint32_t pos) { return wait_or_abort(sh, &sh->kv_full[pos % kSlots], (pos / kSlots) & 1u); };

            const std::false_type full;
            const std::true_type last;
            Item it;
            while (ok && next_item(sh, i, it)) {
                mbar_arrive(&sh->item_empty[i % kItemRing]);
                const int n_x = x == 0 ? it.n_a : it.n_b;
                const int steps = key_steps(visible_keys(p, it, x), n_x);  // of the last tile
                if (!(ok = wait_or_abort(sh, &sh->q_full, i & 1u))) break;
                if (n_x == 0) mbar_arrive(&sh->q_empty);  // this tile never reads the Q buffer of this item
                {
                    const uint32_t kpos = 2 * kt;
                    if (!(ok = slot_full(kpos))) break;
                    if (n_x > 0) {
                        tc_fence_after();
                        const uint64_t kd = k_desc0 + (kpos % kSlots) * kSlotStep;
                        if (n_x > 1)
                            issue_qk(kd, false, full, 8);
                        else
                            issue_qk(kd, false, last, steps);
                        tc_commit(&sh->kv_empty[kpos % kSlots]);
                        if (n_x == 1) tc_commit(&sh->q_empty);
                    } else {
                        mbar_arrive(&sh->kv_empty[kpos % kSlots]);
                    }
                }
                for (int j = 0; ok && j < it.n_kv; ++j) {
                    const uint32_t vpos = 2 * (kt + j) + 1, kpos = vpos + 1;  // ring positions of V(j) and K(j+1)
                    if (!(ok = slot_full(vpos))) break;
                    if (j + 1 < it.n_kv && !(ok = slot_full(kpos))) break;
                    if (j < n_x) {
                        const uint64_t vd = v_desc0 + (vpos % kSlots) * kSlotStep;
                        if (j + 1 < n_x) {
                            if (!(ok = issue_pv(j, vd, full, 8))) break;
                        } else {
                            if (!(ok = issue_pv(j, vd, last, steps))) break;
                            tc_commit(&sh->o_full[x]);
                            tc_commit(&sh->kv_empty[vpos % kSlots]);
                        }
                    } else {
                        mbar_arrive(&sh->kv_empty[vpos % kSlots]);
                    }
                    if (j + 1 < it.n_kv) {
                        if (j + 1 < n_x) {
                            const uint64_t kd = k_desc0 + (kpos % kSlots) * kSlotStep;
                            if (j + 2 < n_x)
                                issue_qk(kd, true, full, 8);
                            else
                                issue_qk(kd, true, last, steps);
                            tc_commit(&sh->kv_empty[kpos % kSlots]);
                            tc_commit(&sh->kv_empty[vpos % kSlots]);
                            if (j + 2 == n_x) tc_commit(&sh->q_empty);  // this tile's last Q.K^T has been issued
                        } else {
                            mbar_arrive(&sh->kv_empty[kpos % kSlots]);
                        }
                    }
                }
                used += n_x > 0 ? 1 : 0;
                kt += it.n_kv;
                ++i;
            }
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
        // ============================ softmax warpgroups ============================
        const int x = (warp - 4) >> 2;              // 0: tile A, 1: tile B
        const int quarter = warp & 3;               // tensor-memory lane quarter this warp may touch
        const int row = quarter * 32 + lane;        // row within the Q tile: a token and a head
        const int tok = row / p.pack.heads, tok_head = row - tok * p.pack.heads;
        const int tok_lo = quarter * 32 / p.pack.heads, tok_hi = (quarter * 32 + 31) / p.pack.heads;  // the warp's tokens
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t t_s = tmem + x * 128 + lane_base;
        const uint32_t t_o = tmem + 256 + x * 128 + lane_base;
        uint32_t tiles = 0;  // tiles finished by this Q tile over all items (barrier phases)
        // Ping-pong between the two softmax warpgroups.  Both tiles' exponentials go through the same four MUFU
        // pipes; if both warpgroups exponentiate at once each takes twice as long and afterwards both tiles' MMAs
        // queue up behind one another.  Inside an item with both tiles active the exponentials therefore alternate
        // A(0) B(0) A(1) B(1) ...: a warpgroup loads its scores and finds the row max while the other one still
        // exponentiates, takes the turn, and hands it over once its last chunk of P is on its way to tensor memory.
        uint32_t turns_seen = 0;  // completions of the other tile's turn barrier this warp has consumed
        uint32_t kt = 0;          // K/V tiles of the items before this one (ring positions)
        bool ok = true;
        Item it;
        for (uint32_t k = 0; ok && next_item(sh, k, it); ++k) {
            const int n_x = x == 0 ? it.n_a : it.n_b;
            const uint32_t kt0 = kt;
            kt += it.n_kv;
            if (n_x == 0) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->item_empty[k % kItemRing]);
                continue;
            }
            // The two tiles take turns, unless tile A has a single K/V tile: then nothing of A could run under B's
            // exponentials, and B's wait is not won back (64 prompts of 20..128 tokens, 32 / 8 heads: 47.9 us without turns,
            // 51.3 with).  With two the turns pay (16 prompts of 256 tokens: 35.7 us without, 34.4 with).
            const bool both = it.n_b > 0 && it.n_a > 1;
            const int q_pos = it.q0 + x * p.pack.dq;      // first token of this Q tile
            const int first_lim = it.prefix + q_pos;      // last key visible to it
            const bool ragged = 16 * key_steps(visible_keys(p, it, x), n_x) + (n_x - 1) * kTileKV > it.len_k;
            const int live = min(p.pack.tokens, it.len - q_pos);  // tokens of the tile in front of the sequence's end
            float m_run = -INFINITY, m_used = -INFINITY, l = 0.f;
            const uint32_t alive = __ballot_sync(0xffffffffu, tok < live);
            // One KV tile of this Q tile.  Tiles whose last key the tile's first row may still see need no mask; the
            // one or two after them (one when the prefix is a multiple of the tile) are masked per element.  The two
            // kinds run in two separate loops so that each loop body is straight-line code.
            auto tile_step = [&](const int j, auto kind) -> bool {
                constexpr bool kDiag = decltype(kind)::value == 1, kDead = decltype(kind)::value == 2;
                if (!wait_or_abort(sh, &sh->s_full[x], tiles & 1u)) return false;
                // A(j) starts after B(j-1); B(j) starts after A(j) while A still has tiles.
                uint64_t* turn_bar = nullptr;
                const uint32_t turn_parity = turns_seen & 1u;
                if (both && (x == 0 ? j >= 1 : j < it.n_a)) {
                    turn_bar = &sh->turn[x ^ 1];
                    ++turns_seen;
                }
                tc_fence_after();
                // keys of this tile that the products go through, and how many of them are the sequence's
                if ((kDiag || kDead) && ragged && j == n_x - 1) {
                    const int through = 16 * key_steps(visible_keys(p, it, x), n_x), own = it.len_k - j * kTileKV;
                    // The last KV tile of the sequence reaches past its last key: those rows of the V tile hold
                    // whatever follows in memory (the next sequence, padding, recycled cache rows).  Their
                    // probabilities are exactly zero, but 0 * NaN or 0 * Inf in the P.V product would still poison the
                    // row, so each thread zeroes "its" row of the V tile before this tile's P is handed over (the
                    // hand-over orders these stores before the MMA that reads them).  Garbage in the K rows is
                    // harmless: those scores are overwritten with -inf by the mask.  This warpgroup trails the MMA
                    // issuer, and the slot cannot be refilled before P.V of this very tile, so the parity wait sees
                    // either "still loading" or "landed", never another tile.  When both Q tiles use the tile both
                    // warpgroups zero it (same bytes, same value).  (Such a tile is always a masked one.)
                    const uint32_t vpos = 2 * (kt0 + j) + 1;
                    if (!wait_or_abort(sh, &sh->kv_full[vpos % kSlots], (vpos / kSlots) & 1u)) return false;
                    if (row >= own && row < through) {
                        // a row is 128 contiguous bytes in each 64-dim panel (the swizzle permutes inside a row)
                        uint8_t* vrow = sKV + (vpos % kSlots) * kTileBytes + row * 128;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            *reinterpret_cast<uint4*>(vrow + c * 16) = make_uint4(0, 0, 0, 0);
                            *reinterpret_cast<uint4*>(vrow + kPanelBytes + c * 16) = make_uint4(0, 0, 0, 0);
                        }
                        fence_proxy_async_smem();  // generic-proxy stores must be visible to the tensor core's reads
                    }
                }
                if constexpr (kDead) {  // nothing but the hand-overs: P and O of these rows may hold anything
                    if (turn_bar != nullptr && !wait_or_abort(sh, turn_bar, turn_parity)) return false;
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (both && (x == 0 || j < it.n_a)) mbar_arrive(&sh->turn[x]);
                        mbar_arrive(&sh->p_full[x][0]);
                        mbar_arrive(&sh->p_full[x][1]);
                    }
                    ++tiles;
                    return true;
                }
                const int lim = first_lim - j * kTileKV;
                if (!softmax_tile<kDiag>(sh, x, t_s, t_o, kDiag ? lim + min(tok, live - 1) : 0, kDiag ? lim + min(tok_lo, live - 1) : 0,
                                         kDiag ? lim + min(tok_hi, live - 1) : 0, j == 0,
                                         (tiles - 1) & 1u, p.scale_log2, alive, m_run, m_used, l, turn_bar, turn_parity,
                                         (both && (x == 0 || j < it.n_a)) ? &sh->turn[x] : nullptr))
                    return false;
                // the turn is handed over by A after each of its tiles, by B after those that followed one of A's
                ++tiles;
                return true;
            };
            const int n_plain = min(n_x, (first_lim + 1) / kTileKV);  // tiles j with j * 128 + 127 <= first_lim
            int j = 0;
            const bool dead = tok_lo >= live;  // the whole warp lies behind the sequence's last row
            if (dead) {
                for (; ok && j < n_x; ++j) ok = tile_step(j, std::integral_constant<int, 2>{});
            } else {
                for (; ok && j < n_plain; ++j) ok = tile_step(j, std::integral_constant<int, 0>{});
                for (; ok && j < n_x; ++j) ok = tile_step(j, std::integral_constant<int, 1>{});
            }
            if (!ok) break;
            // ---- epilogue: O / l -> bf16 -> global, then hand O back to the MMA thread ----
            if (!(ok = wait_or_abort(sh, &sh->o_full[x], (tiles - 1) & 1u))) break;
            tc_fence_after();
            if constexpr (std::is_same<P, SplitParams>::value) {
                if (it.kv0 >= 0) {  // a run of a split item: its O, maximum and sum as they are
                    float* part = p.partials + ((size_t)blockIdx.x * 2 + x) * kPartialFloats;
                    if (!dead) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            uint32_t ov[32];
                            tmem_ld32(t_o + c * 32, ov);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                *reinterpret_cast<uint4*>(part + row * kD + c * 32 + i * 4) =
                                    make_uint4(ov[4 * i], ov[4 * i + 1], ov[4 * i + 2], ov[4 * i + 3]);
                        }
                        part[kTileQ * kD + row] = m_used * p.scale_log2;
                        part[kTileQ * kD + kTileQ + row] = l;
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sh->o_empty[x]);
                        mbar_arrive(&sh->item_empty[k % kItemRing]);
                    }
                    if (x == 0 && both) ok = wait_or_abort(sh, &sh->turn[1], turns_seen++ & 1u);
                    continue;
                }
            }
            const float inv = 1.0f / l;
            const int head = it.head + x * p.pack.dh + tok_head;
            __nv_bfloat16* orow = p.out + ((size_t)(it.seq_start + q_pos + tok) * p.H + head) * kD;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (dead) break;
                uint32_t ov[32];
                tmem_ld32(t_o + c * 32, ov);
                tmem_wait_ld();
                if (tok < live && p.wide) {  // whole sectors: half the store instructions
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t w[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            w[e] = pack_bf16(__uint_as_float(ov[16 * i + 2 * e]) * inv, __uint_as_float(ov[16 * i + 2 * e + 1]) * inv);
                        store_32bytes(orow + c * 32 + i * 16, w);
                    }
                } else if (tok < live) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 w;
                        w.x = pack_bf16(__uint_as_float(ov[8 * i + 0]) * inv, __uint_as_float(ov[8 * i + 1]) * inv);
                        w.y = pack_bf16(__uint_as_float(ov[8 * i + 2]) * inv, __uint_as_float(ov[8 * i + 3]) * inv);
                        w.z = pack_bf16(__uint_as_float(ov[8 * i + 4]) * inv, __uint_as_float(ov[8 * i + 5]) * inv);
                        w.w = pack_bf16(__uint_as_float(ov[8 * i + 6]) * inv, __uint_as_float(ov[8 * i + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = w;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sh->o_empty[x]);
                mbar_arrive(&sh->item_empty[k % kItemRing]);  // only now: the next claim waits for it
            }
            // B's last turn.  Else A, two hand-overs further with the next item's first tile, could lap a warp of B that was
            // held up in front of its last wait (2.7 us would do), and the parity would alias.
            if (x == 0 && both) ok = wait_or_abort(sh, &sh->turn[1], turns_seen++ & 1u);
        }
    }

    // ---- teardown: everyone meets here, then the allocating warp frees tensor memory ----
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && tmem != 0xFFFFFFFFu) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// Puts the runs of split items together: block (item, Q tile, group of 8 rows), thread t owns row t / 16 of the group and
// dims 8 (t % 16) .. + 7.  Latency-bound (the partials are in L2): the maxima of all runs first, then eight runs at a
// time, the ones that are not there included (a loop over the runs, unrolled by four, took the remainder one by one).
constexpr int kCombineThreads = 128;
constexpr int kCombineBatch = 8;
__global__ void __launch_bounds__(kCombineThreads) prefill_combine_kernel(const __grid_constant__ SplitParams p) {
    griddep_wait();
    const int e = blockIdx.x, x = blockIdx.y, row = blockIdx.z * 8 + (threadIdx.x >> 4), c8 = (threadIdx.x & 15) * 8;
    const List list = list_of(p);
    if (e >= items_of(static_cast<const Params&>(p), list) || splits_of(p, list.pairs) == 1) return;
    const Item it = load_item(static_cast<const Params&>(p), list, e);
    const int runs = runs_of(p, p.splits, it.n_a, it.prefix, it.len_k);
    const int tok = row / p.pack.heads, q_pos = it.q0 + x * p.pack.dq + tok;
    if ((x == 0 ? it.n_a : it.n_b) == 0 || runs == 1 || tok >= p.pack.tokens || q_pos >= it.len) return;
    const int head = it.head + x * p.pack.dh + row - tok * p.pack.heads;
    const float* part = p.partials + ((size_t)e * p.splits * 2 + x) * kPartialFloats;
    constexpr size_t kNext = 2 * kPartialFloats;
    float mv[kMaxSplits], m = -INFINITY;
#pragma unroll
    for (int c = 0; c < kMaxSplits; ++c) mv[c] = c < runs ? __ldcg(part + c * kNext + kTileQ * kD + row) : -INFINITY;
#pragma unroll
    for (int c = 0; c < kMaxSplits; ++c) m = fmaxf(m, mv[c]);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, l = 0.f;
#pragma unroll
    for (int c0 = 0; c0 < kMaxSplits; c0 += kCombineBatch) {
        if (c0 >= runs) break;
        float4 a[kCombineBatch], b[kCombineBatch];
        float lv[kCombineBatch];
#pragma unroll
        for (int u = 0; u < kCombineBatch; ++u) {
            const float* q = part + (c0 + u < runs ? c0 + u : 0) * kNext;
            a[u] = __ldcg(reinterpret_cast<const float4*>(q + row * kD + c8));
            b[u] = __ldcg(reinterpret_cast<const float4*>(q + row * kD + c8) + 1);
            lv[u] = __ldcg(q + kTileQ * kD + kTileQ + row);
        }
#pragma unroll
        for (int u = 0; u < kCombineBatch; ++u) {
            if (c0 + u >= runs) break;
            const float f = fast_exp2(mv[c0 + u] - m);
            l += lv[u] * f;
            acc[0] += a[u].x * f, acc[1] += a[u].y * f, acc[2] += a[u].z * f, acc[3] += a[u].w * f;
            acc[4] += b[u].x * f, acc[5] += b[u].y * f, acc[6] += b[u].z * f, acc[7] += b[u].w * f;
        }
    }
    const float inv = 1.0f / l;
    uint4 w;
    w.x = pack_bf16(acc[0] * inv, acc[1] * inv);
    w.y = pack_bf16(acc[2] * inv, acc[3] * inv);
    w.z = pack_bf16(acc[4] * inv, acc[5] * inv);
    w.w = pack_bf16(acc[6] * inv, acc[7] * inv);
    *reinterpret_cast<uint4*>(p.out + ((size_t)(it.seq_start + q_pos) * p.H + head) * kD + c8) = w;
}

// ------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------
static int make_map(CUtensorMap* map, const void* base, int heads, int64_t tokens, int box_heads = 1, int box_tokens = kTileKV) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(NVLLM_B200_EDRIVER, "cuTensorMapEncodeTiled entry point not available");
    // a panel of 64 dims per load: both panels in one load (the half as a fourth dimension) were 1 % slower
    cuuint64_t dims[3] = {(cuuint64_t)kD, (cuuint64_t)heads, (cuuint64_t)tokens};
    cuuint64_t strides[2] = {(cuuint64_t)kD * 2, (cuuint64_t)heads * kD * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_heads, (cuuint32_t)box_tokens};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(NVLLM_B200_EDRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return NVLLM_B200_OK;
}

static int ensure_attr() {
    static std::mutex mu;
    static bool done[64];
    int dev = 0;
    NVLLM_CUDA_OK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        NVLLM_CUDA_OK(cudaFuncSetAttribute(varlen_prefill_kernel<Params>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kSmemBytes));
        NVLLM_CUDA_OK(cudaFuncSetAttribute(varlen_prefill_kernel<SplitParams>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        NVLLM_CUDA_OK(cudaFuncSetAttribute(varlen_prefill_kernel<ShortParams>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        done[dev] = true;
    }
    return NVLLM_B200_OK;
}

static int check_pages(const char* who, int NB, int block_size) {
    if (block_size <= 0 || block_size % kTileKV != 0)
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: block_size %d (must be a multiple of %d)", who, block_size, kTileKV);
    if (NB <= 0) return fail(NVLLM_B200_EINVAL, "%s: NB must be positive", who);
    return NVLLM_B200_OK;
}

static int64_t item_capacity(int64_t T, int B, int span) { return T / span + B + 1; }
static size_t list_bytes(int64_t T, int B, int span) { return ((size_t)(2 * item_capacity(T, B, span) + 1) * 16 + 255) & ~size_t(255); }

// Runs per item: as many as leave one run per SM; 1 where no item can have enough tiles.
static int splits_for(int64_t items, int64_t max_tiles, int sms, int span) {
    if (items <= 0 || 2 * items > sms || max_tiles < kSplitTiles) return 1;
    return (int)std::min<int64_t>(std::min<int64_t>(sms / items, kMaxSplits), max_tiles / min_run(span));
}
// Whether split items are of one Q tile, which has its SM's exponentials to itself and takes no turns, rather than of two.  They are
// twice as many, so where the SMs do not suffice a run has more K/V tiles: worth up to three more where a tile's live rows fill more
// than a warp, none where they do not.  60 new tokens, 32 / 8 heads, behind 3000 cached ones (two / three tiles a run) 24.0 -> 21.3 us,
// behind 6500 (four / six) 29.5 -> 26.0, behind 12 000 (six / eleven, so still of two) 36.0, else 36.3; 16 / 8 heads there 32.7, else 35.6.
static bool lone_tiles(int64_t max_tiles, int splits, int lone_splits, int64_t live_rows) {
    const int more = live_rows > 32 ? 3 : 0;
    return (max_tiles + lone_splits - 1) / lone_splits <= (max_tiles + splits - 1) / splits + more;
}
static size_t partials_bytes(int sms) { return (size_t)sms * 2 * kPartialFloats * 4; }

// Common launcher.  kv_tokens: extent of the token axis of k / v (T for packed tensors, the slot count of the cache).
// sc (may be null): the step's K/V scatter.
static int launch(const char* who, const void* q, const void* k, const void* v, int64_t kv_tokens,
                  const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, const int32_t* block_tables, int MB,
                  int block_size, const int32_t* cu_seqlens_host, void* out, void* workspace, size_t workspace_bytes,
                  int64_t T, int B, int max_seqlen, int H, int KVH, int D, float scale, const Scatter* sc, void* stream) {
    if (T < 0 || B < 0 || H <= 0 || KVH <= 0)
        return fail(NVLLM_B200_EINVAL, "%s: bad size (T=%lld B=%d H=%d KVH=%d)", who, (long long)T, B, H, KVH);
    if (D != kD) return fail(NVLLM_B200_EUNSUPPORTED, "%s: head_dim %d (only 128)", who, D);
    if (H % KVH != 0) return fail(NVLLM_B200_EUNSUPPORTED, "%s: H %d not a multiple of KVH %d", who, H, KVH);
    if (B > 65535) return fail(NVLLM_B200_EUNSUPPORTED, "%s: more than 65535 sequences", who);
    if (T > 0x7fffffffLL || kv_tokens > 0x7fffffffLL)
        return fail(NVLLM_B200_EUNSUPPORTED, "%s: more than 2^31-1 tokens", who);
    if (!(scale > 0.f)) return fail(NVLLM_B200_EINVAL, "%s: scale must be positive", who);
    if (T == 0) return NVLLM_B200_OK;
    const bool scatter = sc && sc->chunks > 0 && sc->num_slots > 0;
    auto scatter_only = [&]() -> int {  // no sequence to attend to: the rows are stored all the same
        return !scatter ? NVLLM_B200_OK
                        : nvllm_b200_store_kvcache(sc->k, sc->v, sc->k_cache, sc->v_cache, sc->slot_mapping, T, KVH, D,
                                                   sc->num_slots, NVLLM_B200_DTYPE_BF16, stream);
    };
    if (B == 0) return scatter_only();
    if (!q || !k || !v || !cu_seqlens_q || !cu_seqlens_k || !out) return fail(NVLLM_B200_EINVAL, "%s: null pointer", who);
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15)
        return fail(NVLLM_B200_EINVAL, "%s: q/k/v/out must be 16-byte aligned", who);
    const int G = H / KVH;
    Pack pack = make_pack(G);
    const size_t need = list_bytes(T, B, pack.span);  // the rest of what is asked for lets items be split
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15))
        return fail(NVLLM_B200_EWORKSPACE, "%s: workspace of %zu bytes required, got %zu", who, need,
                    workspace ? workspace_bytes : (size_t)0);

    ShortParams p;
    int64_t longest = max_seqlen;
    if (cu_seqlens_host) {
        longest = 0;
        for (int b = 0; b < B; ++b) {
            const int64_t len = (int64_t)cu_seqlens_host[b + 1] - cu_seqlens_host[b];
            if (len < 0 || cu_seqlens_host[b + 1] > T)
                return fail(NVLLM_B200_EINVAL, "%s: cu_seqlens_host is not a non-decreasing prefix of T", who);
            if (len > (int64_t)kMaxLevels * kTileKV)
                return fail(NVLLM_B200_EUNSUPPORTED, "%s: sequence of %lld tokens (max %d)", who, (long long)len,
                            kMaxLevels * kTileKV);
            longest = std::max(longest, len);
        }
    } else {
        if (max_seqlen <= 0) return fail(NVLLM_B200_EINVAL, "%s: max_seqlen must be positive", who);
        if (max_seqlen > kMaxLevels * kTileKV)
            return fail(NVLLM_B200_EUNSUPPORTED, "%s: max_seqlen %d (max %d)", who, max_seqlen, kMaxLevels * kTileKV);
    }
    // Upper bound of (sequence, token block) pairs: exact from the host copy of cu_seqlens, else from max_seqlen.
    auto pairs_of = [&](int span) {
        const int64_t cap = item_capacity(T, B, span);
        int64_t n = 0;
        if (cu_seqlens_host) {
            for (int b = 0; b < B; ++b) n += ((int64_t)cu_seqlens_host[b + 1] - cu_seqlens_host[b] + span - 1) / span;
        } else {
            n = (int64_t)B * ((max_seqlen + span - 1) / span);
            // The attention layer's contexts round the longest length up to 8192 at most: prompts beyond it show in T.
            if ((int64_t)B * max_seqlen < T) n = cap;
        }
        return std::min(n, cap);
    };
    int64_t pairs = pairs_of(pack.span);
    if (pairs == 0) return scatter_only();
    if (pairs * KVH * pack.per_kv > 0x7fffffffLL) return fail(NVLLM_B200_EUNSUPPORTED, "%s: grid too large", who);
    const int sms = sm_count();
    const int64_t max_tiles = block_tables ? (int64_t)MB * block_size / kTileKV : (longest + kTileKV - 1) / kTileKV;
    auto splits_with = [&](const Pack& k, int64_t n) {
        const bool room = workspace_bytes >= list_bytes(T, B, k.span) + partials_bytes(sms) && ((uintptr_t)workspace & 255) == 0;
        return room && (block_tables || longest > kWholeKeys) ? splits_for(n * KVH * k.per_kv, max_tiles, sms, k.span) : 1;
    };
    int splits = splits_with(pack, pairs);
    // Longer queries could be split without a prefix, too, and packed keys and keys in pages are to give the same bits.  With queries
    // of at most dq tokens the items have no tile B as it is.
    if (splits > 1 && block_tables && longest < kSplitTiles * kTileKV && longest > pack.dq) {
        const Pack lone = make_pack(G, true);
        const int64_t n = pairs_of(lone.span);
        const int s = splits_with(lone, n);
        if (s > 1 && lone_tiles(max_tiles, splits, s, longest * pack.heads)) pack = lone, pairs = n, splits = s;
    }
    p.pack = pack;
    p.per_pair = KVH * pack.per_kv;

    int rc = ensure_attr();
    if (rc) return rc;
    CUtensorMap tm_q, tm_k, tm_v;
    if ((rc = make_map(&tm_q, q, H, T, pack.heads, pack.tokens))) return rc;
    if ((rc = make_map(&tm_k, k, KVH, kv_tokens))) return rc;
    if ((rc = make_map(&tm_v, v, KVH, kv_tokens))) return rc;

    p.items = (const int4*)workspace;
    p.cu_seqlens = cu_seqlens_q;
    p.B = B;
    p.block_tables = block_tables;
    p.MB = MB;
    p.block_size = block_size;
    p.out = (__nv_bfloat16*)out;
    p.H = H;
    p.G = G;
    p.wide = ((uintptr_t)out & 31) == 0;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.scatter = Scatter{};
    int ctas = p.item_ctas = (int)std::min<int64_t>(pairs * p.per_pair, sms);

    // A short list known to the host (and nothing for the plan kernel to check on the device) needs no plan kernel, and
    // the scatter, where SMs are left, goes with the launch.  Elsewhere the scatter is a launch of its own: on a warp of the
    // attention CTAs it slowed them by as much as it took (power and issue slots).
    const bool brief = splits == 1 && cu_seqlens_host && !block_tables && cu_seqlens_k == cu_seqlens_q &&
                       B <= kShortSequences && pairs <= kShortBlocks && pairs * p.per_pair <= sms;
    if (scatter) {
        const int64_t blocks = (store_blocks_for(sc->chunks) + kThreads / kStoreThreads - 1) / (kThreads / kStoreThreads);
        if (brief && ctas + blocks <= sms) {
            p.scatter = *sc;
            ctas += (int)blocks;
        } else if ((rc = scatter_only())) {
            return rc;
        }
    }

    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    if (!brief) {
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(kPlanThreads);
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, prefill_plan_kernel, cu_seqlens_q, cu_seqlens_k, block_tables ? 1 : 0, B,
                                         (int4*)workspace, (int)item_capacity(T, B, pack.span), pack.span, p.per_pair, KVH, ctas,
                                         scatter && pdl_enabled() ? 1 : 0));
    }
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    if (splits > 1) {
        SplitParams sp;
        static_cast<Params&>(sp) = p;
        sp.partials = (float*)((uint8_t*)workspace + list_bytes(T, B, pack.span));
        sp.splits = splits;
        sp.ctas = (int)(pairs * p.per_pair * splits);
        cfg.gridDim = dim3((unsigned)sp.ctas);
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, varlen_prefill_kernel<SplitParams>, tm_q, tm_k, tm_v, sp));
        cfg.gridDim = dim3((unsigned)(pairs * p.per_pair), 2, kTileQ / 8);
        cfg.blockDim = dim3(kCombineThreads);
        cfg.dynamicSmemBytes = 0;
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, prefill_combine_kernel, sp));
    } else if (brief)
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, varlen_prefill_kernel<ShortParams>, tm_q, tm_k, tm_v, p));
    else
        NVLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, varlen_prefill_kernel<Params>, tm_q, tm_k, tm_v, (const Params&)p));
    return NVLLM_B200_OK;
}

}  // namespace prefill

int read_prefill_flags(int* out) {
    NVLLM_CUDA_OK(cudaMemcpyFromSymbol(out, prefill::g_error_flag, sizeof(int)));
    return NVLLM_B200_OK;
}
int clear_prefill_flags() {
    const int zero = 0;
    NVLLM_CUDA_OK(cudaMemcpyToSymbol(prefill::g_error_flag, &zero, sizeof(int)));
    return NVLLM_B200_OK;
}
}  // namespace nvllm

extern "C" size_t nvllm_b200_varlen_prefill_workspace_bytes(int64_t T, int B, int H, int KVH, int D) {
    using namespace nvllm;
    using namespace nvllm::prefill;
    (void)D;
    if (T < 0 || B < 0) return 256;
    if (H <= 0 || KVH <= 0 || H % KVH != 0) return list_bytes(T, B, 1);
    const Pack pack = make_pack(H / KVH);
    size_t n = list_bytes(T, B, pack.span);
    // room for the partial results of split items where so few items are possible
    const int64_t blocks = std::max<int64_t>((T + pack.span - 1) / pack.span, B), per_pair = (int64_t)KVH * pack.per_kv;
    if (2 * blocks * per_pair <= sm_count())
        n = list_bytes(T, B, make_pack(H / KVH, true).span) + partials_bytes(sm_count());
    return n;
}

extern "C" int nvllm_b200_varlen_prefill(const void* q, const void* k, const void* v, const int32_t* cu_seqlens_q,
                                         const int32_t* cu_seqlens_k, const int32_t* cu_seqlens_host, void* out,
                                         void* workspace, size_t workspace_bytes, int64_t T, int B, int max_seqlen,
                                         int H, int KVH, int D, float scale, void* stream) {
    // packed keys/values lie beside the queries (k, v are [T, KVH, 128] like q): cu_seqlens_k must equal
    // cu_seqlens_q, which the plan kernel checks on the device
    return nvllm::prefill::launch("varlen_prefill", q, k, v, T, cu_seqlens_q, cu_seqlens_k, nullptr, 0, 0,
                                  cu_seqlens_host, out, workspace, workspace_bytes, T, B, max_seqlen, H, KVH, D, scale,
                                  nullptr, stream);
}

extern "C" int nvllm_b200_paged_prefill(const void* q, const void* k_cache, const void* v_cache,
                                        const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k,
                                        const int32_t* block_tables, const int32_t* cu_seqlens_q_host, void* out,
                                        void* workspace, size_t workspace_bytes, int64_t T, int B, int max_seqlen_q,
                                        int H, int KVH, int D, int NB, int block_size, int MB, float scale,
                                        void* stream) {
    using namespace nvllm;
    if (!block_tables || MB <= 0) return fail(NVLLM_B200_EINVAL, "paged_prefill: block_tables required");
    int rc = prefill::check_pages("paged_prefill", NB, block_size);
    if (rc) return rc;
    return prefill::launch("paged_prefill", q, k_cache, v_cache, (int64_t)NB * block_size, cu_seqlens_q, cu_seqlens_k,
                           block_tables, MB, block_size, cu_seqlens_q_host, out, workspace, workspace_bytes, T, B,
                           max_seqlen_q, H, KVH, D, scale, nullptr, stream);
}

extern "C" int nvllm_b200_prefill_step(const void* q, const void* k, const void* v, void* k_cache, void* v_cache,
                                       const int32_t* slot_mapping, const int32_t* cu_seqlens_q,
                                       const int32_t* cu_seqlens_k, const int32_t* block_tables,
                                       const int32_t* cu_seqlens_q_host, void* out, void* workspace,
                                       size_t workspace_bytes, int64_t T, int B, int max_seqlen_q, int H, int KVH, int D,
                                       int NB, int block_size, int MB, float scale, void* stream) {
    using namespace nvllm;
    const char* who = "prefill_step";
    if (T < 0 || KVH <= 0 || NB <= 0 || block_size <= 0 || (block_tables && MB <= 0))
        return fail(NVLLM_B200_EINVAL, "%s: bad size (T=%lld KVH=%d NB=%d block=%d MB=%d)", who, (long long)T, KVH, NB,
                    block_size, MB);
    if (D != prefill::kD) return fail(NVLLM_B200_EUNSUPPORTED, "%s: head_dim %d (only 128)", who, D);
    if (T == 0) return NVLLM_B200_OK;
    if (!k || !v || !k_cache || !v_cache || !slot_mapping) return fail(NVLLM_B200_EINVAL, "%s: null pointer", who);
    if (((uintptr_t)k | (uintptr_t)v | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15)
        return fail(NVLLM_B200_EINVAL, "%s: k/v and caches must be 16-byte aligned", who);
    int rc = block_tables ? prefill::check_pages(who, NB, block_size) : NVLLM_B200_OK;
    if (rc) return rc;
    const int row_chunks = KVH * D / 8;
    const int64_t num_slots = (int64_t)NB * block_size;
    const Scatter sc = {(const __nv_bfloat16*)k, (const __nv_bfloat16*)v, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache,
                        slot_mapping, T * row_chunks, row_chunks, num_slots};
    return prefill::launch(who, q, block_tables ? k_cache : k, block_tables ? v_cache : v, block_tables ? num_slots : T,
                           cu_seqlens_q, cu_seqlens_k, block_tables, MB, block_size, cu_seqlens_q_host, out, workspace,
                           workspace_bytes, T, B, max_seqlen_q, H, KVH, D, scale, &sc, stream);
}
