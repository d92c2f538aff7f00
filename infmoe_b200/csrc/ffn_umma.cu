// Grouped expert FFN on the Blackwell tensor cores (sm_100a): tcgen05.mma with
// TMEM accumulators, operands staged by TMA, split-operand error compensation so
// the products keep FP32 accuracy.
//
// Replaces, for all experts at once, the per-expert sequence of
// T5FFLayer::run (plugin/sublayers/T5FFLayer.cc:112-138):
//   cublasSgemm_v2 x2 (wi_0, wi_1) -> fused_gelu_dot_gpu -> cudaMemcpyAsync D2D -> cublasSgemm_v2 (beta = 1)
//
// Two launches of one kernel template (the weights are the M-side operand):
//   EPI_GELU_PAIR  g = gelu(h wi_0^T) * (h wi_1^T)   K = d_model, weight rows = 2 * d_ff
//                  (rows of wi_0 and wi_1 are stored interleaved: row 2f = wi_0[f], row 2f+1 = wi_1[f],
//                   so both halves of the gate land in neighbouring TMEM lanes of ONE accumulator)
//   EPI_RESIDUAL   y = x + g wo^T                     K = d_ff,    weight rows = d_model
//
// Orientation.  Weight rows sit on the MMA's M side (always a full 128-row
// tile), the tokens of one expert on the N side (any multiple of 16 up to
// NMAX).  An expert with 139 tokens therefore costs one N=144 tile instead of
// two 128-token tiles, and a decode step with 1..64 tokens runs N=16..64 MMAs.
// The accumulator is D^T: TMEM lane = weight row, TMEM column = token.
//
// Split operands.  Both operands are pairs of FP16 values, x 2^s = hi + lo (common.cuh, split_f16): hi has 11
// significant bits and lo the next 11 or 12, so the pair holds the FP32 value to its last bit or the one before it.
// w * x = lo(w) hi(x) + hi(w) lo(x) + hi(w) hi(x) + (a term below 2^-22): three kind::f16 products, six K = 16 MMAs
// per k block of 32.  s is a power of two per weight row (its largest value lands in [2^14, 2^15), chosen when the
// weights are laid out) and per token row (from the row itself for h, from a bound that cannot be exceeded for g,
// see g_exponent); the epilogues multiply the sums by 2^-s, which is exact.  Powers of two per column, which cancel between
// the operands, even the rows out beforehand (rows.cu, SplitExpert).
// The pair takes the four bytes of the FP32 value in HBM, L2 and shared memory, and nothing has to be converted on
// the way to the tensor cores.  What it replaced, a TF32 head product with BF16 corrections of weights that four
// warps split between shared memory and TMEM, took 8 MMAs and about 1000 cycles per k block (of 144 tokens), held
// by the conversion and by 106 KB of shared-memory traffic; this form moves about 80 KB and needs 6.  Relative error
// against 64 bits (layer output, d_model 4096): 1.4e-6, was 2.3e-6.
//
// Chunked accumulation.  The tensor core adds into its FP32 accumulator with
// truncation, not round-to-nearest: measured on B200, one accumulator carried
// over K = 1024..2048 drifts by about 1.5e-5 relative, and the drift grows
// linearly with the number of MMAs.  So a TMEM accumulator only ever holds the
// sum of one chunk of 8 k blocks (48 MMAs, the first one overwriting); the
// accumulate warps add each finished chunk into a running sum in registers with
// round-to-nearest adds, in ascending k.  That order is the same for every tile,
// whatever the launch, so a token's result does not depend on its neighbours.
//
// Pipeline per CTA (persistent, one CTA per SM, 20 warps):
//   warp 0        TMA producer: a stage is one weight tile (16 KB) and the token tile of the same k block
//   warp 1        MMA issuer (and owner of the TMEM allocation): one commit per k block frees the stage, one per chunk
//                 hands its accumulator to the accumulate warps.  Chunks rotate over as many accumulators as fit into
//                 TMEM at the width of the launch's widest token tile (2 at 192 columns, 4 at 128, at most 8)
//   warp 2        walks the schedule and lists the CTA's items (tiles, or parts of cut ones) for the others, up to four ahead
//   warp 3        fetches what the epilogue needs of an item (scales of its rows, output rows, mix coefficients)
//   warps 4..19   accumulate + epilogue: tcgen05.ld the chunk (one TMEM lane quarter and a quarter of the
//                 columns per warp, 4 of 16 to 48 of 192), add into registers; after the last chunk gelu*dot and its
//                 split (lane pairs exchange a and b by shuffle) or residual add.  The epilogue is a chain of
//                 shuffles, loads and stores, so warps in flight set its speed, and with K = 1024 or less it sets the
//                 kernel's: 8 -> 16 warps (and 8 residual values in flight per thread instead of 16, which spilled)
//                 took 8 experts x 256 x 1024 with 16384 tokens from 296 to 209 us per layer, three layers of 8 x 1024 x
//                 4096 with 4096 tokens from 1446 to 1284, 777 tokens x 12 x 1000 x 2724 from 154 to 132
//
// Pairs (CTAS = 2, a cluster of two).  Both CTAs walk the same items; tile rows 0..127 belong to the first one, 128..255
// to the second.  Each fetches its own weight tile and its half of the token rows, counting on the first one's barrier;
// the first one's issuer runs the MMAs for both (M = 256) and its commits arrive in both; both CTAs' accumulate warps
// hand the accumulator back to it.
//
// Tiles are (expert, 128-row weight block, token chunk); the list is derived in
// the kernel from offset[E+1], so no host synchronisation is needed.
//
// The last, partly filled round of tiles is cut along K.  With fewer tiles left than CTAs, the tiles' chunks are
// dealt out evenly over all CTAs.  A CTA that holds part of a tile stores its chunk sums (the holder of the first
// chunks one running sum), and the warp that finds itself the last one on its part of the tile adds them up in
// ascending k and runs the epilogue.  Nobody waits, and the additions are those of an uncut tile, so the bits are too.
// One token through one expert of 4096 x 10240 (32 tiles of 320 k blocks on 148 SMs): second GEMM 158 -> 58 us.
//
// Layer times beside a step are those before and after that step, in the code of its time: they do not add up to today's.
//
// Every mbarrier wait is bounded: on expiry the CTA raises STATUS_WAIT_TIMEOUT, lets
// copies in flight land, frees its TMEM and returns.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace infmoe {

namespace {

constexpr int UMMA_M = 128;
constexpr int MAX_EXPERTS = 1024;
constexpr unsigned long long WAIT_LIMIT_NS = 4000000000ull;  // 4 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Same with a suspend-time hint: the thread may sleep in hardware for up to `ns` nanoseconds and is woken when
// the phase completes, instead of polling: polling warps take issue slots from the working warps of their scheduler.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when the wait was abandoned (limit reached here or in another role).
// The common case, a barrier that is already complete, is a single try_wait (about 17 cycles).
static __device__ __forceinline__ bool mbar_wait_limited(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                               unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    while (true) {
        for (int i = 0; i < 16; ++i)
            if (mbar_try_wait_sleep(bar, parity, 100000u)) return true;   // sleeps, up to 0.1 ms at a time
        if (*abort_flag) return false;
        if (global_ns() - t0 > limit_ns) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return mbar_wait_limited(bar, parity, abort_flag, WAIT_LIMIT_NS);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_slow(bar, parity, abort_flag);
}

// L2 policies of a load: weights that one tile alone reads give way first, so that streaming them does not push out what
// the passes come back to (activations, chunk sums, centroids, and the kernels' code).  Layer, us: one token 32 x 4096 x 10240
// 118.7 -> 108.8, 777 tokens 12 x 1000 x 2724 113 -> 104, 2500 tokens 16 x 512 x 2048 131 -> 118.
__device__ __forceinline__ uint64_t l2_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_normal() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
// True for one thread of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T: FP16 operands, both K-major in shared memory, K = 16 per instruction.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same over a pair of CTAs (M = 256): each CTA's shared memory holds 128 rows of A and half the rows of B, each
// CTA's tensor memory 128 rows of D.  Issued by the first CTA of the pair.
__device__ __forceinline__ void umma_f16_ss_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int CTAS>
__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if (CTAS == 1) umma_f16_ss(d, a, b, idesc, accumulate);
    else umma_f16_ss_pair(d, a, b, idesc, accumulate);
}
// Arrives on the barrier at this offset in both CTAs of the pair once all MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"((uint16_t)3)
        : "memory");
}
// Address of a shared-memory location of this CTA in the first CTA of the pair.
__device__ __forceinline__ uint32_t leader_addr(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A load into this CTA's shared memory that counts on a barrier of the pair's first CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair_hint(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                      uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], "
        "[%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
        : "memory");
}
// Arrives on the mbarrier once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

constexpr int BK = 32;                     // k block: 32 values = one 128-byte swizzled row (32 x hi, 32 x lo)
constexpr int ROW_BYTES = BK * 4;

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzled rows (8-row groups of 1024 bytes).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);    // start address
    d |= (uint64_t)1 << 16;                       // leading byte offset: not used by swizzled K-major layouts
    d |= (uint64_t)((8 * ROW_BYTES) >> 4) << 32;  // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                       // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                       // SWIZZLE_128B
    return d;
}

// Instruction descriptor: FP16 operands (format 0), FP32 accumulate, both operands K-major, M = m, N = n.
__device__ __forceinline__ uint32_t make_idesc(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

enum { EPI_GELU_PAIR = 0, EPI_RESIDUAL = 1 };

constexpr int TMA_WARP = 0;
constexpr int MMA_WARP = 1;                           // issues all MMAs; owns the TMEM allocation
constexpr int ITEM_WARP = 2;                          // walks the schedule ahead of the others
constexpr int COLUMN_WARP = 3;                        // fetches what the epilogue needs of each tile
constexpr int EPI_WARP0 = 4;
constexpr int EPI_GROUPS = 4;                         // warps per TMEM lane quarter
constexpr int EPI_WARPS = 4 * EPI_GROUPS;
constexpr int GEMM_THREADS = (EPI_WARP0 + EPI_WARPS) * 32;
constexpr int TMEM_COLS = 512;
constexpr int CHUNK_BLOCKS = 8;                       // k blocks (of 6 MMAs) an accumulator takes between two drains
constexpr int SUM_FLIGHT = 8;                         // chunk sums a thread fetches at a time (narrow tiles)
constexpr int W_TILE = UMMA_M * ROW_BYTES;            // 16 KB of weights per k block

template <int NMAX, int STAGES, int CTAS>
struct Cfg {
    static constexpr int STAGE = W_TILE + NMAX / CTAS * ROW_BYTES;  // weight tile, then this CTA's part of the token tile
    static constexpr int SMEM = STAGES * STAGE + 1024;              // + slack for 1024-byte alignment
    static constexpr int MAX_ACC = 8;                                // accumulators, at most
    static constexpr int SLICES = (NMAX / EPI_GROUPS + 15) / 16;     // 16-column slices owned by one epilogue thread
    static constexpr int N_STEP = 16 * CTAS;                        // token tiles are padded to a multiple of this
    static_assert(NMAX % N_STEP == 0 && 2 * NMAX <= TMEM_COLS, "token chunk");
    static_assert((NMAX / CTAS * ROW_BYTES) % 1024 == 0, "tiles must keep 1024-byte alignment");
};

struct GemmArgs {
    const int* offset;          // [E+1] first routed row of each expert
    const int* gate;            // [tokens] experts of the tokens, to count instead of reading offset[] (NULL: read it)
    int tokens;
    int early;                  // GELU_PAIR: what offset or gate points to is complete when the kernel starts
    const int* slot_of_expert;  // expert -> weight slot (NULL: identity)
    int E, e_begin, e_end;      // experts [e_begin, e_end) are processed
    int M_total;                // weight rows: 2 * d_ff (wi_0 / wi_1 rows interleaved) or d_model
    int K;
    const float* w;             // weight plane: per slot the tiles, then the rows' 2^-s (see split_plane_elems)
    size_t w_stride;            // floats per slot
    const int* bound;           // w of g_exponent: first slot ...
    size_t bound_stride;        // ... and words from one slot to the next
    const float2* row_info;     // [T] of the h rows: 2^-s and log2 of the squared norm
    void* out_pack;             // GELU_PAIR: packed plane of g
    float* out;                 // RESIDUAL: y [T][M_total]
    const float* resid;         // RESIDUAL: the rows the experts were applied to, indexed like the output: row
                                // out_pos[j] (or j) of x [rows][M_total]; no routed copy of x is needed
    const int* out_pos;         // RESIDUAL: row j is written to row out_pos[j] of y (NULL: row j), i.e. the combine
                                // step moe_expert_gather (plugin/cuda/moe.cu:89-96) fused into the epilogue
    const float* mix_score;     // RESIDUAL: routed scores for the base_layer output mix (NULL: no mix)
    const unsigned long long* out_row_ptr;   // RESIDUAL: address of output row i (i = out_pos[j] or j) instead of
                                             // y + i * M_total; the rows may live in another GPU's memory
    float4* part;               // chunk sums of cut tiles: blocks of [part_cols / 4][128 rows] float4 (NULL: nothing is cut)
    int part_blocks, part_cols;
    int* part_count;            // [gridDim][EPI_WARPS] chunks of a cut tile stored so far; zero between launches
    int* status;
};

// Tensor maps of the packed token plane, one per box height 16, 32, ... 192 rows: a tile's load fetches exactly
// the rows its MMAs read (n_pad), not the largest tile's worth.
constexpr int TOKEN_BOXES = 12;
struct TokenMaps {
    CUtensorMap pk[TOKEN_BOXES];
};

struct TileInfo {
    int expert, slot, mb, row0, n_tok, n_pad;
};

// An entry of the list that the item warp writes and the others read: chunks [c0, c1) of a tile (c1 = 0: no more items).
// tail: index among the cut tiles (-1: this CTA holds the whole tile), prefix: chunks that the tile's first holder sums up;
// alone: the expert's weights are read by this token tile only.
struct __align__(16) ListItem {
    int c0, c1, tail, prefix;
    int row0, n_tok, n_pad, slot;
    int mb, alone, unused[2];
};
constexpr int ITEM_SLOTS = 4;

template <int NMAX, int STEP>
__device__ __forceinline__ void chunking(int cnt, int& nch, int& csz) {
    nch = (cnt + NMAX - 1) / NMAX;
    csz = nch ? (((cnt + nch - 1) / nch + STEP - 1) & ~(STEP - 1)) : 0;  // balanced chunks, multiple of STEP, <= NMAX
}

// Tiles are listed by expert in order of falling token count (s_order: list position -> expert, s_prefix: first
// tile of each list position), so the long tiles of the busiest experts are handed out first and the short ones
// fill the end of the schedule.
template <int NMAX, int STEP>
__device__ __forceinline__ TileInfo decode_tile(int tile, const int* s_prefix, const short* s_order, const int* s_beg,
                                                const int* s_cnt, const GemmArgs& a) {
    int lo = 0, hi = a.E - 1;  // last list position with s_prefix[.] <= tile
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_prefix[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    TileInfo t;
    const int ex = s_order[lo];
    t.expert = ex;
    t.slot = a.slot_of_expert ? a.slot_of_expert[ex] : ex;
    const int beg = s_beg[ex], cnt = s_cnt[ex];
    int nch, csz;
    chunking<NMAX, STEP>(cnt, nch, csz);
    const int local = tile - s_prefix[lo];
    t.mb = local / nch;                 // chunk-minor: CTAs working side by side share the weight tile in L2
    const int c = local % nch;
    t.row0 = beg + c * csz;
    t.n_tok = min(csz, beg + cnt - t.row0);
    t.n_pad = (t.n_tok + STEP - 1) & ~(STEP - 1);
    return t;
}

// A CTA's share of the work, walked identically by every role.  Whole rounds of gridDim tiles come first: the CTAs
// walk the (sorted) list forwards in even rounds and backwards in odd ones, so that over two rounds every CTA gets
// one tile from each end of a stretch.  The R tiles left after the last whole round are cut into chunk units and dealt
// out evenly when that pays: an uncut tail lasts one tile (m chunks), a cut one R m / G chunks plus storing and
// re-reading the chunk sums, which is worth about two chunks (measured on narrow tiles, the same for wide ones by assumption), and
// where the chunk sums fit into the scratch (ffn_umma_part_bytes).  A CTA whose share spans two tiles stores, fences and counts
// twice, about as long as a chunk and a half; where shares that end with their tile are at most that much longer, they are
// taken.  Layer, us: 2500 tokens 16 x 512 x 2048 104 -> 90, one token 32 x 4096 x 10240 109 -> 105.
struct Item {
    int tile;
    int c0, c1;        // chunks [c0, c1) of the tile
    int tail;          // index among the cut tiles, -1: this CTA holds the whole tile
};
template <int CTAS>
struct Schedule {
    int m, full, rounds, round;      // chunks of a tile, whole rounds, whole tiles of this CTA, those it has taken
    int per, u, hi;                  // chunks of a holder's share where no share spans two tiles, else 0; the units it has left
    static __device__ __forceinline__ int ctas() { return (int)gridDim.x / CTAS; }
    static __device__ __forceinline__ int first_unit(int b, int units, int cuts) { return (int)((long long)b * units / cuts); }
    __device__ __forceinline__ int whole_tile(int r) const {
        const int b = (int)blockIdx.x / CTAS;
        return r * ctas() + ((r & 1) ? ctas() - 1 - b : b);
    }
    __device__ __forceinline__ Schedule(int total, int KB, const GemmArgs& a) {
        const int G = ctas(), b = (int)blockIdx.x / CTAS;
        m = (KB + CHUNK_BLOCKS - 1) / CHUNK_BLOCKS;
        full = total / G;
        rounds = full;
        round = per = u = hi = 0;
        const int R = total - full * G, units = R * m;
        if (R == 0) return;
        if (!a.part || (long long)(G - R) * m < 2ll * G || (long long)units * CTAS > a.part_blocks) {
            if (whole_tile(full) < total) ++rounds;
            return;
        }
        per = (m + G / R - 1) / (G / R);
        if (2 * per * G <= 2 * units + 3 * G) {
            const int holders = (m + per - 1) / per;
            if (b < R * holders) {
                u = b / holders * m + b % holders * per;
                hi = min(u + per, (b / holders + 1) * m);
            }
        } else {
            per = 0;
            const int cuts = min(G, units);
            if (b < cuts) {
                u = first_unit(b, units, cuts);
                hi = first_unit(b + 1, units, cuts);
            }
        }
    }
    __device__ __forceinline__ bool next(Item& it) {
        if (round < rounds) {
            it.tile = whole_tile(round);
            it.c0 = 0;
            it.c1 = m;
            it.tail = -1;
            ++round;
            return true;
        }
        if (u >= hi) return false;
        const int t = u / m;
        it.tile = full * ctas() + t;
        it.c0 = u - t * m;
        it.c1 = min(m, hi - t * m);
        it.tail = (it.c0 == 0 && it.c1 == m) ? -1 : t;
        u = t * m + it.c1;
        return true;
    }
    // chunks of cut tile t, of `total` tiles, that its first holder sums up in registers
    __device__ __forceinline__ int prefix_chunks(int t, int total) const {
        if (per) return per;
        const int units = (total - full * ctas()) * m, cuts = min(ctas(), units);
        const long long u0 = (long long)t * m;
        const int b = (int)(((u0 + 1) * cuts - 1) / units);     // holder of unit u0
        return min(m, (int)(first_unit(b + 1, units, cuts) - u0));
    }
};

template <int EPI, int NMAX, int STAGES, int CTAS>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
ffn_umma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokenMaps token_maps,
                const GemmArgs args) {
    using C = Cfg<NMAX, STAGES, CTAS>;
    extern __shared__ uint8_t smem_raw[];
    // k block `it` (counted over all items of the CTA) uses stage it % STAGES; chunks rotate over the accumulators
    __shared__ __align__(8) uint64_t s_full[STAGES];        // TMA -> MMA: stage filled
    __shared__ __align__(8) uint64_t s_empty[STAGES];       // MMA -> TMA: stage consumed
    __shared__ __align__(8) uint64_t s_acc_full[C::MAX_ACC];   // MMA -> accumulate warps: chunk done
    __shared__ __align__(8) uint64_t s_acc_empty[C::MAX_ACC];  // accumulate warps -> MMA: chunk read out
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ int s_widest;
    __shared__ int s_prefix[MAX_EXPERTS + 1];
    __shared__ int s_cnt[MAX_EXPERTS];
    __shared__ int s_beg[MAX_EXPERTS];
    __shared__ short s_order[MAX_EXPERTS];
    // the next items, and what the epilogue needs of each: two words per column (2^-s of the token row and 2^s of g, or 2^-s of
    // the row of g and the output row), the mix coefficients, 2^-s of the weight rows
    __shared__ ListItem s_item[ITEM_SLOTS];
    __shared__ __align__(16) float2 s_col[ITEM_SLOTS][NMAX];
    __shared__ float s_mix[EPI == EPI_RESIDUAL ? ITEM_SLOTS : 1][NMAX];
    __shared__ __align__(16) float s_winv[ITEM_SLOTS][UMMA_M];
    __shared__ __align__(8) uint64_t s_item_full[ITEM_SLOTS];   // item warp -> all others
    __shared__ __align__(8) uint64_t s_col_full[ITEM_SLOTS];    // column warp -> accumulate warps
    __shared__ __align__(8) uint64_t s_item_empty[ITEM_SLOTS];  // all others -> item warp

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int MB1 = (args.M_total + UMMA_M - 1) / UMMA_M;    // 128-row weight blocks
    const int MB = (MB1 + CTAS - 1) / CTAS;                  // of which a tile has CTAS
    uint32_t rank = 0;
    if (CTAS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int KB = (args.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&s_full[s]), 1);
            mbar_init(smem_u32(&s_empty[s]), 1);
        }
        for (int b = 0; b < C::MAX_ACC; ++b) {
            mbar_init(smem_u32(&s_acc_full[b]), 1);
            mbar_init(smem_u32(&s_acc_empty[b]), EPI_WARPS * CTAS);
        }
        for (int i = 0; i < ITEM_SLOTS; ++i) {      // an item's readers: producer, column warp, issuer, accumulate warps
            mbar_init(smem_u32(&s_item_full[i]), 1);
            mbar_init(smem_u32(&s_col_full[i]), 32);
            mbar_init(smem_u32(&s_item_empty[i]), 2 + (rank == 0 ? 1 : 0) + EPI_WARPS);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        if (CTAS == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                         "r"((uint32_t)TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                         "r"((uint32_t)TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    // Work before the wait.  The scatter kernels and the first GEMM let their successor's blocks start only after their own
    // wait.  So when a block of the second GEMM starts, everything before the first one is complete, and it can read
    // offset[], make its schedule and fetch weights while the first one's last tiles are still running; what the first one
    // writes it touches after its own wait, further down.  In the same way the first GEMM (`early`) starts while the
    // scatter is still running: offset[] is complete when a kernel of its own has made it, and the gates are when the scatter
    // makes offset[] itself.
    // Layer, us, second GEMM: 32 tokens 64 x 256 24.5 -> 22.3, one token 4096 x 10240 138.5 -> 133.7, 777 x 12 x 1000 x 2724
    // 124 -> 120; first GEMM and scatter: one token 132.5 -> 125, 777 tokens 117 -> 112, 2500 x 16 x 512 x 2048 140 -> 130.
    const bool early = EPI == EPI_RESIDUAL || args.early;
    if (!early) pdl_wait();
    if (EPI == EPI_RESIDUAL || !early) pdl_trigger();

    // ---- tile schedule: experts by falling token count, exclusive prefix of their tiles ---------
    if (EPI == EPI_GELU_PAIR && args.gate) {
        for (int e = threadIdx.x; e < args.E; e += GEMM_THREADS) s_cnt[e] = 0;
        __syncthreads();
        for (int t0 = threadIdx.x; t0 < args.tokens; t0 += 8 * GEMM_THREADS) {
            int e[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) e[i] = t0 + i * GEMM_THREADS < args.tokens ? __ldcg(args.gate + t0 + i * GEMM_THREADS) : -1;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (e[i] >= 0 && e[i] < args.E) atomicAdd(&s_cnt[e[i]], 1);
        }
        __syncthreads();
        if (warp == 2) {
            int carry = 0;
            for (int e0 = 0; e0 < args.E; e0 += 32) {
                const int e = e0 + lane, c = e < args.E ? s_cnt[e] : 0;
                int incl = c;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int n = __shfl_up_sync(0xffffffffu, incl, off);
                    if (lane >= off) incl += n;
                }
                if (e < args.E) s_beg[e] = carry + incl - c;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
    } else {
        for (int e = threadIdx.x; e < args.E; e += GEMM_THREADS) {
            const int beg = __ldcg(args.offset + e);
            s_beg[e] = beg;
            s_cnt[e] = (e >= args.e_begin && e < args.e_end) ? __ldcg(args.offset + e + 1) - beg : 0;
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < args.E; e += GEMM_THREADS) {
        const int c = s_cnt[e];
        int rank = 0;   // experts that come before e: more tokens, or as many and a lower index
        for (int o = 0; o < args.E; ++o) {
            const int co = s_cnt[o];
            rank += (co > c || (co == c && o < e)) ? 1 : 0;
        }
        s_order[rank] = (short)e;
    }
    __syncthreads();
    if (warp == 0) {
        int carry = 0, widest = 16;
        for (int e0 = 0; e0 < args.E; e0 += 32) {
            const int e = e0 + lane;   // list position
            int nt = 0;
            if (e < args.E) {
                int nch, csz;
                chunking<NMAX, C::N_STEP>(s_cnt[s_order[e]], nch, csz);
                nt = nch * MB;
                widest = max(widest, csz);
            }
            int incl = nt;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += n;
            }
            if (e < args.E) s_prefix[e] = carry + incl - nt;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        widest = __reduce_max_sync(0xffffffffu, widest);
        if (lane == 0) {
            s_prefix[args.E] = carry;
            s_widest = widest;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CTAS > 1) cluster_sync();    // the barriers of both CTAs are ready
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    // as many accumulators as fit beside one another at the width of the widest token tile
    const uint32_t acc_stride = (uint32_t)s_widest, nacc = min((uint32_t)C::MAX_ACC, (uint32_t)TMEM_COLS / acc_stride);
    volatile int* abort_flag = &s_abort;
    const int m_chunks = (KB + CHUNK_BLOCKS - 1) / CHUNK_BLOCKS;
    // A reader's place in the list of items.
    struct Place {
        uint32_t slot = 0, phase = 0;
        __device__ __forceinline__ void advance() {
            if (++slot == ITEM_SLOTS) {
                slot = 0;
                phase ^= 1;
            }
        }
    };

    // every thread of an early first GEMM passes here once, its producer when it has fetched its first weights
    const auto wait_then_trigger = [&]() {
        if (EPI == EPI_GELU_PAIR && early) {
            pdl_wait();
            pdl_trigger();
        }
    };
    if (warp == TMA_WARP) {
        // ================= TMA producer =================
        if (lane == 0) {
            uint32_t it = 0, ahead = 0;    // ahead: k blocks whose weights were fetched before the wait
            bool ok = true, waited = !early;
            const uint64_t evict_first = l2_evict_first(), evict_normal = l2_evict_normal();
            const auto wait = [&]() {
                if (EPI == EPI_RESIDUAL) pdl_wait();
                wait_then_trigger();
                waited = true;
            };
            for (Place at; ok; at.advance()) {
                if (!mbar_wait(smem_u32(&s_item_full[at.slot]), at.phase, abort_flag)) break;
                const ListItem t = s_item[at.slot];
                if (t.c1 == 0) break;
                mbar_arrive(smem_u32(&s_item_empty[at.slot]));
                // a box of n_pad token rows (rows past the chunk's tokens belong to the next expert or are
                // zero-filled past the end; they only feed accumulator columns that are never stored)
                const int n_own = t.n_pad / CTAS;
                const CUtensorMap* map_pk = &token_maps.pk[(n_own >> 4) - 1];
                const uint32_t bytes = W_TILE + n_own * ROW_BYTES;
                // a second CTA past the last weight block loads that block again and drops the result
                const int mb = min(t.mb * CTAS + (int)rank, MB1 - 1);
                const int w_row0 = (int)(args.w_stride / BK) * t.slot + mb * KB * UMMA_M;
                const int kb_begin = t.c0 * CHUNK_BLOCKS, kb_end = min(KB, t.c1 * CHUNK_BLOCKS);
                const uint64_t policy = t.alone ? evict_first : evict_normal;
                const auto fetch_weights = [&](uint32_t s, int kb) {
                    const uint32_t bar = smem_u32(&s_full[s]), dst = ring + s * C::STAGE;
                    if (CTAS == 1) {
                        mbar_expect_tx(bar, bytes);
                        tma_load_2d_hint(dst, &map_w, bar, 0, w_row0 + kb * UMMA_M, policy);
                    } else {
                        if (rank == 0) mbar_expect_tx(bar, CTAS * bytes);
                        tma_load_2d_pair_hint(dst, &map_w, leader_addr(bar), 0, w_row0 + kb * UMMA_M, policy);
                    }
                };
                const auto fetch_tokens = [&](uint32_t s, int kb) {
                    const uint32_t bar = smem_u32(&s_full[s]), dst = ring + s * C::STAGE + W_TILE;
                    if (CTAS == 1) tma_load_2d(dst, map_pk, bar, kb * 2 * BK, t.row0);
                    else tma_load_2d_pair(dst, map_pk, leader_addr(bar), kb * 2 * BK, t.row0 + (int)rank * n_own);
                };
                if (!waited) {
                    for (int kb = kb_begin; kb < kb_end && ahead < STAGES; ++kb, ++ahead) fetch_weights(ahead, kb);
                    asm volatile("prefetch.tensormap [%0];" ::"l"(map_pk) : "memory");
                    wait();
                }
                for (int kb = kb_begin; kb < kb_end; ++kb, ++it) {
                    const uint32_t s = it % STAGES;
                    if (it >= ahead) {
                        if (!mbar_wait(smem_u32(&s_empty[s]), ((it / STAGES) & 1) ^ 1, abort_flag)) { ok = false; break; }
                        fetch_weights(s, kb);
                    }
                    fetch_tokens(s, kb);
                }
            }
            if (!waited) wait();
        } else {
            wait_then_trigger();
        }
    } else if (warp == MMA_WARP) {
        // ================= MMA issuer =================
        // One elected thread runs the whole loop (elect.sync tells the compiler so).  With the warp running it and lane 0
        // issuing, the operands of every MMA had to be moved to uniform registers behind a divergent branch: ~148
        // cycles per MMA whatever its N, which held a decode step of 27 experts at 1694 us of first GEMM where the
        // same bytes stream in 1269.  Elected: 1259 us (7.2 TB/s); 4096 tokens 2780 -> 2383.
        wait_then_trigger();
        if (rank == 0 && elect_one()) {
            auto commit = [](uint32_t bar) {
                if (CTAS == 1) umma_commit(bar);
                else umma_commit_pair(bar);
            };
            uint32_t it = 0, acc = 0, acc_phase = 0;
            bool ok = true;
            for (Place at; ok; at.advance()) {
                if (!mbar_wait(smem_u32(&s_item_full[at.slot]), at.phase, abort_flag)) break;
                const int c0 = s_item[at.slot].c0, c1 = s_item[at.slot].c1;
                const uint32_t idesc = make_idesc(UMMA_M * CTAS, s_item[at.slot].n_pad);
                if (c1 == 0) break;
                mbar_arrive(smem_u32(&s_item_empty[at.slot]));
                for (int c = c0; ok && c < c1; ++c) {
                    const uint32_t d = tmem_base + acc * acc_stride;
                    if (!mbar_wait(smem_u32(&s_acc_empty[acc]), acc_phase ^ 1, abort_flag)) { ok = false; break; }
                    const int kb0 = c * CHUNK_BLOCKS, kb_end = min(KB, kb0 + CHUNK_BLOCKS);
                    for (int kb = kb0; kb < kb_end; ++kb, ++it) {
                        const uint32_t s = it % STAGES;
                        if (!mbar_wait(smem_u32(&s_full[s]), (it / STAGES) & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                        const uint64_t dw = make_smem_desc(ring + s * C::STAGE), dx = make_smem_desc(ring + s * C::STAGE + W_TILE);
                        // In a row hi is bytes 0..63, lo bytes 64..127; 32 bytes along K = 2 units of the descriptor
                        // address.  Corrections first (small terms).
                        umma_f16<CTAS>(d, dw + 4, dx, idesc, kb == kb0 ? 0u : 1u);
                        umma_f16<CTAS>(d, dw + 6, dx + 2, idesc, 1u);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            umma_f16<CTAS>(d, dw + 2 * j, dx + 4 + 2 * j, idesc, 1u);
                            umma_f16<CTAS>(d, dw + 2 * j, dx + 2 * j, idesc, 1u);
                        }
                        commit(smem_u32(&s_empty[s]));
                        if (kb + 1 == kb_end) commit(smem_u32(&s_acc_full[acc]));
                    }
                    if (++acc == nacc) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp >= EPI_WARP0) {
        // ================= accumulate + epilogue =================
        // Each chunk is accumulated in TMEM (its first MMA overwrites the accumulator) and added here, with
        // round-to-nearest adds in ascending k, to a running sum in registers; then the accumulator goes back to the
        // MMA issuer.
        const int q = warp & 3;                 // TMEM lane quarter this warp may access
        const int group = (warp - EPI_WARP0) >> 2;   // columns [group, group + 1) / EPI_GROUPS of the tile
        const uint32_t tlane = tmem_base + ((uint32_t)(q * 32) << 16);
        uint32_t acc = 0, acc_phase = 0;
        bool ok = true;
        if (EPI == EPI_RESIDUAL) pdl_wait();
        wait_then_trigger();
        for (Place at; ok; at.advance()) {
            // the warp stays converged for the .aligned TMEM instructions, also when a wait is abandoned
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_item_full[at.slot]), at.phase, abort_flag))) break;
            const ListItem& t = s_item[at.slot];     // read where it is used: a copy would take registers from the sums
            if (t.c1 == 0) break;
            const auto done_with_item = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_item_empty[at.slot]));
            };
            const int width = t.n_pad / EPI_GROUPS, col0 = group * width;    // this warp's columns; a multiple of 4
            float sum[C::SLICES][16];
#pragma unroll
            for (int i = 0; i < C::SLICES; ++i)
#pragma unroll
                for (int c = 0; c < 16; ++c) sum[i][c] = 0.f;
            const int row = q * 32 + lane;      // row of the tile this thread works on
            const int mb = t.mb * CTAS + (int)rank, m = mb * UMMA_M + row;
            const int block = (args.part_cols >> 2) * UMMA_M;   // float4 per block of chunk sums
            const auto part_of_tile = [&]() { return args.part + ((size_t)t.tail * CTAS + rank) * m_chunks * (size_t)block + row; };
            auto store_block = [&](int c) {     // sum[][] -> block of chunk c
                float4* const dst = part_of_tile() + (size_t)c * block;
#pragma unroll
                for (int i = 0; i < C::SLICES; ++i)
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        if (16 * i + 4 * v >= width) continue;
                        __stcg(dst + ((col0 >> 2) + 4 * i + v) * UMMA_M,
                               make_float4(sum[i][4 * v], sum[i][4 * v + 1], sum[i][4 * v + 2], sum[i][4 * v + 3]));
                    }
            };
            for (int c = t.c0; c < t.c1; ++c) {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_acc_full[acc]), acc_phase, abort_flag))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < C::SLICES; ++i) {
                    if (16 * i >= width) continue;       // uniform across the warp
                    const uint32_t at = tlane + acc * acc_stride + col0 + 16 * i;
                    uint32_t r[16];
                    if (16 * i + 16 <= width) {
                        tmem_ld16(at, r);
                    } else {
#pragma unroll
                        for (int x = 0; x < 16; ++x) r[x] = 0;
#pragma unroll
                        for (int v = 0; v < 3; ++v)
                            if (16 * i + 4 * v < width) tmem_ld4(at + 4 * v, r + 4 * v);
                    }
                    tmem_ld_wait();
#pragma unroll
                    for (int x = 0; x < 16; ++x) sum[i][x] = __fadd_rn(sum[i][x], __uint_as_float(r[x]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CTAS == 1) mbar_arrive(smem_u32(&s_acc_empty[acc]));
                    else mbar_arrive_cluster(leader_addr(smem_u32(&s_acc_empty[acc])));
                }
                if (++acc == nacc) {
                    acc = 0;
                    acc_phase ^= 1;
                }
                if (t.tail >= 0 && (t.c0 > 0 || c + 1 == t.c1)) {
                    store_block(c);
#pragma unroll
                    for (int i = 0; i < C::SLICES; ++i)
#pragma unroll
                        for (int x = 0; x < 16; ++x) sum[i][x] = 0.f;
                }
            }
            if (!ok) break;
            if (t.tail >= 0) {
                // Each warp of the CTAs that share a tile owns the same rows and columns of it; the last of them to
                // arrive here finishes them.
                __threadfence();
                __syncwarp();
                int done = 0;
                int* const counter = args.part_count + (t.tail * CTAS + rank) * EPI_WARPS + (warp - EPI_WARP0);
                if (lane == 0) {
                    done = atomicAdd(counter, t.c1 - t.c0) + t.c1 - t.c0;
                    if (done == m_chunks) *counter = 0;    // everybody has arrived; ready for the next launch
                    __threadfence();
                }
                done = __shfl_sync(0xffffffffu, done, 0);
                __syncwarp();    // orders lane 0's fence before the other lanes' reads of the sums; a shuffle does not
                if (done != m_chunks) {
                    done_with_item();
                    continue;
                }
                const int first = t.prefix - 1;
                if constexpr (C::SLICES == 1) {
                    // few columns: one of the thread's float4 at a time, SUM_FLIGHT chunks of it on their way together (a trip is
                    // 1.4 us; one token through 4096 x 10240 has 40 chunk sums per tile).  Eight: ten spill, which every drain pays
                    // for (decode of 8 tokens 533 -> 547 us, 128 tokens 11 x 512 x 1408 42.2 -> 45.0)
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        if (4 * v >= width) continue;
                        const float4* src = part_of_tile() + ((col0 >> 2) + v) * UMMA_M;
                        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                        for (int c0 = first; c0 < m_chunks; c0 += SUM_FLIGHT) {
                            float4 x[SUM_FLIGHT];
#pragma unroll
                            for (int c = 0; c < SUM_FLIGHT; ++c)
                                if (c0 + c < m_chunks) x[c] = __ldcg(src + (size_t)(c0 + c) * block);
#pragma unroll
                            for (int c = 0; c < SUM_FLIGHT; ++c) {
                                if (c0 + c >= m_chunks) break;
                                y.x = __fadd_rn(y.x, x[c].x);
                                y.y = __fadd_rn(y.y, x[c].y);
                                y.z = __fadd_rn(y.z, x[c].z);
                                y.w = __fadd_rn(y.w, x[c].w);
                            }
                        }
                        sum[0][4 * v] = y.x;
                        sum[0][4 * v + 1] = y.y;
                        sum[0][4 * v + 2] = y.z;
                        sum[0][4 * v + 3] = y.w;
                    }
                } else {
                    // eight float4 in flight; more of them spill
#pragma unroll
                    for (int i = 0; i < C::SLICES; ++i) {
                        if (16 * i >= width) continue;
                        const float4* src = part_of_tile() + ((col0 >> 2) + 4 * i) * UMMA_M;
#pragma unroll 2
                        for (int c = first; c < m_chunks; ++c) {
#pragma unroll
                            for (int v = 0; v < 4; ++v) {
                                if (16 * i + 4 * v >= width) continue;
                                const float4 x = __ldcg(src + (size_t)c * block + v * UMMA_M);
                                sum[i][4 * v] = __fadd_rn(sum[i][4 * v], x.x);
                                sum[i][4 * v + 1] = __fadd_rn(sum[i][4 * v + 1], x.y);
                                sum[i][4 * v + 2] = __fadd_rn(sum[i][4 * v + 2], x.z);
                                sum[i][4 * v + 3] = __fadd_rn(sum[i][4 * v + 3], x.w);
                            }
                        }
                    }
                }
            }
            if (mb >= MB1) {
                done_with_item();
                continue;
            }
            const bool m_ok = m < args.M_total;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_col_full[at.slot]), at.phase, abort_flag))) break;
            const float w_inv = s_winv[at.slot][row];
            const float2* const s_tab = &s_col[at.slot][col0];      // this warp's columns
            const float* const s_alpha = &s_mix[EPI == EPI_RESIDUAL ? at.slot : 0][col0];
            if constexpr (EPI == EPI_GELU_PAIR) {
                // Even weight row = wi_0 (a), odd row = wi_1 (b) of the same d_ff index f, so a lane pair holds (a, b) of f for
                // all token columns.  The pair splits the columns: the even lane takes the even ones, the odd lane the odd
                // ones; one shuffle per column pair hands each lane the half it lacks, and every gelu is evaluated once.
                // Packed plane: neighbouring f (lanes two apart, same column) exchange their halves so that every lane stores
                // one 32-bit word, even f the pair of hi, odd f the pair of lo.  The plane is zero padded to whole groups of
                // 32 (weight rows past the matrix are zero, so those values are 0).
                const int F = args.M_total >> 1, f = m >> 1, odd = lane & 1;
                const uint32_t pitch = (uint32_t)pack_pitch(F), halves = (f & 1) ? 0x3276u : 0x5410u;
                uint16_t* const out = reinterpret_cast<uint16_t*>(args.out_pack) + (size_t)(t.row0 + col0 + odd) * pitch +
                                      (size_t)(f >> 5) * 64 + (f & 31) + ((f & 1) ? 31 : 0);
                const int end = f < ((F + 31) & ~31) ? min(t.n_tok - col0, width) - odd : 0;    // columns this lane stores
                // Eight columns at a time, every step for all of them before the next: one chain of shared-memory read, shuffle,
                // exponential, reciprocal, conversions, shuffle and store is some 300 cycles, and a store keeps the
                // compiler from starting the next one above it.  128 columns: 9.3 -> 6.8 thousand cycles.  (Conversions and
                // the second shuffle for two columns at a time changed nothing.)
#pragma unroll
                for (int i = 0; i < 2 * C::SLICES; ++i) {
                    if (8 * i >= width) continue;     // uniform across the warp
                    float* const v = &sum[i >> 1][8 * (i & 1)];
                    const float4* const cols = reinterpret_cast<const float4*>(s_tab + 8 * i);
                    float a[4], b[4];
                    uint32_t hl[4], nb[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 col = cols[c];
                        const float v0 = unscale(v[2 * c], w_inv, col.x), v1 = unscale(v[2 * c + 1], w_inv, col.z);
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
                        a[c] = odd ? got : v0;
                        b[c] = odd ? v1 : got;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 col = cols[c];
                        hl[c] = split_f16(gelu_dot_fast(a[c], b[c]) * (odd ? col.w : col.y));
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) nb[c] = __shfl_xor_sync(0xffffffffu, hl[c], 2);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (8 * i + 2 * c < end)
                            *reinterpret_cast<uint32_t*>(out + (size_t)(8 * i + 2 * c) * pitch) = __byte_perm(hl[c], nb[c], halves);
                }
            } else {
#pragma unroll
                for (int i = 0; i < C::SLICES; ++i) {
                    if (16 * i >= width) continue;     // uniform across the warp
                    unsigned long long lane_ptr = 0;   // address of the output row of column 16 i + (lane & 15)
                    if (args.out_row_ptr && 16 * i + (lane & 15) < min(width, t.n_tok - col0))
                        lane_ptr = args.out_row_ptr[__float_as_int(s_tab[16 * i + (lane & 15)].y)];
                    // The residual values of eight columns are fetched first, all in flight together: issued
                    // one by one between the stores (which may alias them as far as the compiler knows) each would
                    // cost a trip to L2, and the next tile's first chunk would wait.
#pragma unroll
                    for (int c0 = 0; c0 < 16; c0 += 8) {
                        if (16 * i + c0 >= width) continue;
                        const int end = m_ok ? min(t.n_tok - col0, width) - (16 * i + c0) : 0;    // columns of these eight to store
                        int r[8];
                        float y[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            r[c] = __float_as_int(s_tab[16 * i + c0 + c].y);
                            y[c] = c < end ? args.resid[(size_t)r[c] * (size_t)args.M_total + (size_t)m] : 0.f;
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            const float x = y[c];
                            y[c] = __fadd_rn(x, unscale(sum[i][c0 + c], w_inv, s_tab[16 * i + c0 + c].x));
                            if (args.mix_score) {
                                const float alpha = s_alpha[16 * i + c0 + c];
                                y[c] = mix_value(alpha, 1.0f - alpha, y[c], x);
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            float* out = args.out + (size_t)r[c] * (size_t)args.M_total;
                            if (args.out_row_ptr) out = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, lane_ptr, c0 + c));
                            if (c < end) out[m] = y[c];
                        }
                    }
                }
            }
            done_with_item();
        }
    } else if (warp == ITEM_WARP) {
        // ================= list of items =================
        // The schedule and the place of a tile (searches, divisions) take one to two thousand cycles, and every role took them
        // at each tile, the issuer and the accumulate warps while nothing else went on in their part.  Layer, us, with the
        // column warp: 4096 tokens 8 x 1024 x 4096 331 -> 321, 16384 tokens 64 x 1024 x 4096 1481 -> 1432, 32 tokens 4 x 64 x 256,
        // where the list is only a detour, 18.1 -> 18.8.
        Schedule<CTAS> sched(s_prefix[args.E], KB, args);
        Place at;
        bool more = true, first = true;
        while (more) {
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_item_empty[at.slot]), at.phase ^ 1, abort_flag))) break;
            Item item;
            more = sched.next(item);
            ListItem e = {};
            if (more) {
                const TileInfo t = decode_tile<NMAX, C::N_STEP>(item.tile, s_prefix, s_order, s_beg, s_cnt, args);
                e.c0 = item.c0;
                e.c1 = item.c1;
                e.tail = item.tail;
                e.prefix = item.tail >= 0 ? sched.prefix_chunks(item.tail, s_prefix[args.E]) : 0;
                e.row0 = t.row0;
                e.n_tok = t.n_tok;
                e.n_pad = t.n_pad;
                e.slot = t.slot;
                e.mb = t.mb;
                e.alone = s_cnt[t.expert] <= NMAX ? 1 : 0;
            }
            if (lane == 0) {
                s_item[at.slot] = e;
                mbar_arrive(smem_u32(&s_item_full[at.slot]));
            }
            __syncwarp();
            at.advance();
            if (first) wait_then_trigger();
            first = false;
        }
    } else if (warp == COLUMN_WARP) {
        // ================= columns of the items =================
        // Fetched by the accumulate warps, slice by slice when the sums were complete, these were a chain of trips to memory:
        // 4096 tokens 8 x 1024 x 4096 355 -> 340 us, 2500 tokens 16 x 512 x 2048 118 -> 110.
        if (EPI == EPI_RESIDUAL) pdl_wait();
        wait_then_trigger();
        for (Place at;; at.advance()) {
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_item_full[at.slot]), at.phase, abort_flag))) break;
            const ListItem t = s_item[at.slot];
            if (t.c1 == 0) break;
            const int mb = t.mb * CTAS + (int)rank;
            if (mb < MB1) {
                // 2^-s of the weight rows (padding rows have one too)
                const float* const scales = args.w + (size_t)t.slot * args.w_stride + (size_t)MB1 * KB * (UMMA_M * BK);
                const float4 inv = __ldg(reinterpret_cast<const float4*>(scales + mb * UMMA_M) + lane);
                const float bound = (float)__ldg(args.bound + (size_t)t.slot * args.bound_stride);
                for (int c = lane; c < t.n_pad; c += 32) {
                    const bool ok = c < t.n_tok;
                    const float2 info = ok ? args.row_info[t.row0 + c] : make_float2(1.f, 0.f);
                    const int g_exp = g_exponent(info.y, bound);
                    if (EPI == EPI_GELU_PAIR) {
                        s_col[at.slot][c] = make_float2(info.x, exp2_int(g_exp));
                    } else {
                        const int r = ok && args.out_pos ? args.out_pos[t.row0 + c] : t.row0 + c;
                        s_col[at.slot][c] = make_float2(exp2_int(-g_exp), __int_as_float(r));
                        if (args.mix_score && ok)
                            s_mix[EPI == EPI_RESIDUAL ? at.slot : 0][c] = mix_alpha(args.mix_score[t.row0 + c]);
                    }
                }
                reinterpret_cast<float4*>(s_winv[at.slot])[lane] = inv;
            }
            mbar_arrive(smem_u32(&s_col_full[at.slot]));
            __syncwarp();      // the slot is used again only after this phase of its columns, also where nobody waits for them
            if (lane == 0) mbar_arrive(smem_u32(&s_item_empty[at.slot]));
        }
    }

    // ---- teardown ---------------------------------------------------------------------------
    tc_fence_before();
    __syncthreads();
    if (s_abort) {
        if (threadIdx.x == 0 && args.status) atomicOr(args.status, STATUS_WAIT_TIMEOUT);
        // let copies that were already issued land before the shared memory is released
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (CTAS > 1) cluster_sync();    // nobody touches the other CTA's shared or tensor memory any more
    if (warp == MMA_WARP) {
        tc_fence_after();
        if (CTAS == 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                         : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                         : "memory");
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// map over a row-major matrix [rows][K] of FP32 (or, for the packed token plane, 16-bit) elements; box = 128 bytes x
// box_rows, 128-byte swizzle
int make_map(CUtensorMap* map, const void* base, uint64_t K, uint64_t rows, int box_rows, bool half = false) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return INFMOE_ERR_CUDA;
    }
    const uint64_t esz = half ? 2 : 4;
    cuuint64_t dims[2] = {K, rows};
    cuuint64_t strides[1] = {K * esz};
    cuuint32_t box[2] = {(cuuint32_t)(ROW_BYTES / esz), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                          const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with %d (K=%llu rows=%llu box=%dx%d)", (int)r,
                  (unsigned long long)K, (unsigned long long)rows, BK, box_rows);
        return INFMOE_ERR_CUDA;
    }
    return INFMOE_OK;
}

// The token maps of a call depend only on the plane pointer, K and the row count, which repeat from call
// to call (same workspace): the last few sets are kept per host thread instead of being encoded again.
int token_maps(TokenMaps* out, const void* pack, int K, long long T) {
    struct Entry {
        const void* pack = nullptr;
        int K = 0;
        long long T = 0;
        TokenMaps maps;
    };
    static thread_local Entry cache[4];
    static thread_local int next = 0;
    for (const Entry& e : cache)
        if (e.pack == pack && e.K == K && e.T == T) {
            *out = e.maps;
            return INFMOE_OK;
        }
    Entry& e = cache[next];
    next = (next + 1) % 4;
    e.pack = nullptr;   // stays invalid if an encode fails
    for (int b = 0; b < TOKEN_BOXES; ++b)
        INFMOE_TRY(make_map(&e.maps.pk[b], pack, pack_pitch(K), (uint64_t)T, 16 * (b + 1), true));
    e.pack = pack;
    e.K = K;
    e.T = T;
    *out = e.maps;
    return INFMOE_OK;
}

template <int EPI, int NMAX, int STAGES, int CTAS>
int launch_one(GemmArgs args, long long T, int slots, const void* tokens, size_t part_bytes, int num_ctas,
               cudaStream_t stream) {
    using C = Cfg<NMAX, STAGES, CTAS>;
    static_assert(C::SMEM + 26 * 1024 <= 227 * 1024, "shared-memory ring too large");
    static_assert(NMAX / CTAS <= 16 * TOKEN_BOXES, "a token tile needs a tensor map of its height");
    args.part_cols = (int)(T < NMAX ? (T + C::N_STEP - 1) / C::N_STEP * C::N_STEP : NMAX);
    const size_t blocks = part_bytes / ((size_t)args.part_cols * UMMA_M * sizeof(float));
    args.part_blocks = (int)(blocks < 0x7fffffff ? blocks : 0x7fffffff);
    CUtensorMap map_w;
    TokenMaps tm;
    // weights: the plane as a [rows][32] matrix of 128-byte rows, one 16 KB tile per box
    INFMOE_TRY(make_map(&map_w, args.w, BK, (uint64_t)slots * (args.w_stride / BK), UMMA_M));
    INFMOE_TRY(token_maps(&tm, tokens, args.K, T));
    auto kern = ffn_umma_kernel<EPI, NMAX, STAGES, CTAS>;
    INFMOE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    INFMOE_CUDA_TRY(launch_chained(kern, (unsigned)(num_ctas / CTAS * CTAS), GEMM_THREADS, C::SMEM, CTAS, stream, map_w, tm, args));
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

// One warp waits on a barrier that nothing ever completes, through the same bounded wait the GEMM roles use, with
// a caller-chosen limit: the way to see the expiry path (flag, status bit, orderly return) without a real stall.
__global__ void wait_probe_kernel(unsigned long long limit_ns, int* status, unsigned long long* waited_ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int s_abort;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const unsigned long long t0 = global_ns();
    const bool done = mbar_wait_limited(smem_u32(&bar), 0, &s_abort, limit_ns);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!done && s_abort) atomicOr(status, STATUS_WAIT_TIMEOUT);
        *waited_ns = global_ns() - t0;
    }
}

}  // namespace

// Tensor map over a row-major FP32 matrix [rows][K] with boxes of 32 floats x box_rows rows and the 128-byte swizzle
// (for the other kernels of the library; K * 4 and the base address must be multiples of 16 bytes).
int make_f32_row_map(CUtensorMap* map, const void* base, long long K, long long rows, int box_rows) {
    return make_map(map, base, (uint64_t)K, (uint64_t)rows, box_rows);
}

int launch_wait_probe(unsigned long long limit_ns, int* status, unsigned long long* waited_ns, cudaStream_t stream) {
    wait_probe_kernel<<<1, 32, 0, stream>>>(limit_ns, status, waited_ns);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

bool ffn_umma_supported(int D, int F, int E) {
    return D % 4 == 0 && F % 4 == 0 && D >= 8 && F >= 8 && E <= MAX_EXPERTS;
}

// Grouped FFN over experts [e_begin, e_end); T rows in expert-contiguous order.
int launch_ffn_umma(const FfnUmma& f, long long T, int D, int F, int E, int e_begin, int e_end, int num_sms,
                    cudaStream_t stream, cudaEvent_t mid_event) {
    if (T == 0 || e_begin >= e_end) return INFMOE_OK;
    if (!ffn_umma_supported(D, F, E)) {
        set_error("ffn_umma: unsupported shape D=%d F=%d E=%d", D, F, E);
        return INFMOE_ERR_UNSUPPORTED;
    }
    static_assert(FFN_COUNTERS == FFN_CTAS * EPI_WARPS, "counters of the cut tiles");
    if (num_sms > FFN_CTAS) num_sms = FFN_CTAS;
    GemmArgs a1{};
    a1.offset = f.offset;
    a1.gate = f.gate;
    a1.tokens = (int)T;
    a1.early = f.early ? 1 : 0;
    a1.slot_of_expert = f.slot_of_expert;
    a1.E = E;
    a1.e_begin = e_begin;
    a1.e_end = e_end;
    a1.M_total = 2 * F;
    a1.K = D;
    a1.w = f.w01;
    a1.w_stride = split_plane_elems(2 * F, D);
    a1.bound = reinterpret_cast<const int*>(f.w01 + split_range_at(2 * F, D));
    a1.bound_stride = a1.w_stride;
    a1.row_info = reinterpret_cast<const float2*>(f.row_info);
    a1.out_pack = f.g;
    a1.part = reinterpret_cast<float4*>(f.part);
    a1.part_count = f.part_count;
    a1.status = f.status;
    GemmArgs a2 = a1;
    a2.M_total = D;
    a2.K = F;
    a2.w = f.wo;
    a2.w_stride = split_plane_elems(D, F);
    a2.out_pack = nullptr;
    a2.out = f.out;
    a2.resid = f.resid;
    a2.out_pos = f.out_pos;
    a2.mix_score = f.mix_score;
    a2.out_row_ptr = f.out_row_ptr;
    // Token chunk, ring and CTAs per tile.
    //   few tokens per expert   64 columns, so that the ring holds more, smaller stages: 128 KB of weights on their way
    //                           per SM instead of 80 KB
    //   K from 2048             pairs of CTAs on tiles of 256 weight rows (cta_group::2).  Each CTA fetches and holds half of
    //                           the token tile, so shared memory takes 63 instead of 78 KB of traffic per k block of 144
    //                           tokens and L2 half the token reads; where the GPU is at its power cap that is time.
    //                           Layer, us, one CTA / pairs: 4096 tokens 32 x 4096 x 10240 4173 / 3900, 16384 tokens
    //                           12485 / 11651; second GEMM of 777 x 12 x 1000 x 2724 (K = 2724) 52 / 47.  Token tiles of a pair
    //                           are padded to 32; 18, 24, 33, 40 tokens per expert, 32 x 2048 x 4096: 565 / 557, 567 / 570,
    //                           579 / 585, 583 / 591, 32 x 4096 x 10240 20 and 36: 2389 / 2366, 2440 / 2466; the most it costs is
    //                           what 20 tokens cost at 64 x 2048 x 2048, 600 / 632.  With one 128-row weight block, of which
    //                           the second CTA has none: 4 x 128 x 4096, 1024 tokens 86 / 83, 8 x 128 x 2048, 4096 108 / 113
    //   shorter K               one CTA: the epilogue, not the MMAs, is in front, and from 144 columns on there are only two
    //                           accumulators to compute the next tile's chunks into meanwhile; first GEMM, us: K = 1024, 16
    //                           experts x 4096, 1000 tokens 104 / 112, K = 680, 6 experts, 4640 tokens 65 / 80
    const bool small = T <= 64 || T <= 16ll * (e_end - e_begin);
    const auto pick = [&](auto epi, const GemmArgs& a, const void* tokens) -> int {
        constexpr int EPI = decltype(epi)::value;
        if (small) return launch_one<EPI, 64, 8, 1>(a, T, f.slots, tokens, f.part_bytes, num_sms, stream);
        if (a.K >= 2048) return launch_one<EPI, 192, 7, 2>(a, T, f.slots, tokens, f.part_bytes, num_sms, stream);
        return launch_one<EPI, 192, 5, 1>(a, T, f.slots, tokens, f.part_bytes, num_sms, stream);
    };
    INFMOE_TRY(pick(std::integral_constant<int, EPI_GELU_PAIR>(), a1, f.h));
    if (mid_event) INFMOE_CUDA_TRY(cudaEventRecord(mid_event, stream));
    INFMOE_TRY(pick(std::integral_constant<int, EPI_RESIDUAL>(), a2, f.g));
    return INFMOE_OK;
}

// Room for the chunk sums of cut tiles: what the cut tail of either GEMM can need (fewer than FFN_CTAS tiles of up to
// max(D, F) / 256 chunks), up to 64 MB; beyond that the tail stays uncut.  That is no rare case: from 192 tokens on a block
// is 192 columns wide whatever the tiles are, 682 of them fit, one for each chunk, cut tile and CTA of a pair, and the second GEMM
// of most batches wants more: 4096 tokens, 8 x 1024 x 4096, 704 (its second round of tiles has 22 of 74 pairs at work),
// 777 tokens, 12 x 1000 x 2724, 1056.
size_t ffn_umma_part_bytes(long long T, int D, int F) {
    const int K = D > F ? D : F;
    const size_t chunks = (size_t)((K + BK - 1) / BK + CHUNK_BLOCKS - 1) / CHUNK_BLOCKS;
    const size_t cols = (size_t)(T < 192 ? (T + 31) / 32 * 32 : 192);    // the widest token tile
    const size_t need = (size_t)FFN_CTAS * chunks * cols * UMMA_M * sizeof(float);
    return need < (64u << 20) ? need : (size_t)(64u << 20);
}

}  // namespace infmoe
