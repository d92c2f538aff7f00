// Exact-FP32 grouped expert FFN on CUDA cores.  This is the path for shapes the
// tensor-core kernels cannot take (d_model or d_ff not divisible by 4) and the
// cross-check used while validating the tcgen05 kernels on the device.  It is not a
// fallback for a missing GPU: it runs on the same device from the same buffers.
//
// Math (T5FFLayer::run, plugin/sublayers/T5FFLayer.cc:112-138), per expert e on
// its rows [offset[e], offset[e+1]):
//   g = gelu(h wi_0^T) * (h wi_1^T)
//   y = x + g wo^T
// Activations are FP32 rows padded with zeros to a multiple of 32 values; weights are raw FP32 in tiles of 128 rows x
// 32 values (launch_retile), wi_0 and wi_1 sharing one matrix with interleaved rows (row 2f = wi_0[f], row
// 2f+1 = wi_1[f]).  So whatever the widths are, every row of a k block is 128 aligned bytes.
//
// Bound by shared-memory reads for many rows per expert, by the number of CTAs for few.  With few, a cluster of up to four CTAs
// computes 16 RI token rows x 32 outputs, each CTA a part of the k blocks, and adds the parts up through distributed shared
// memory; with many, one CTA takes the parts one after the other, with the same additions (launch_ffn_simt).  A thread has RI x 4
// (x 2 when both matrices are multiplied) outputs.  K blocks of 32 are fetched by 16-byte cp.async into two
// buffers.  Both operands stay row-major in shared memory at a pitch of 36 floats, and a thread reads
// four k of a row at a time: 4 + 8 128-bit loads for 128 multiply-adds, without bank conflicts (the eight weight rows a
// warp reads at once start 4 banks apart; token rows are broadcasts).  Every output is up to four chains of FMAs in
// ascending k, cut by K alone, so a row's result does not depend on the other rows of the call.
// Layer of 300 tokens, 6 experts, 510 x 1022: 423 -> 103 us (it was 64 x 64 tiles of scalar loads, one buffer, TF32 head
// and tail planes added on the fly), 88 with the dispatch and scatter in one kernel, 67 with the clusters: 96 to 192 CTAs of
// one chain each had left two or three of four schedulers of an SM without a warp, now 384 to 768 are in flight, six to an
// SM (at 80 registers; five, at 96, left 28 of 768 CTAs for a second wave: 66.8 -> 65.6).  Half the threads with twice the
// rows each, 16 loads for 256 multiply-adds, took 2.6 us longer.  The shorter chains also halve the error against 64 bits,
// 4.6e-7 -> 2.4e-7.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace infmoe {

namespace {

constexpr int SIMT_THREADS = 128;
constexpr int TN = 32;       // outputs per CTA
constexpr int TK = 32;       // one k block of the weight tiles
constexpr int PITCH = TK + 4;
constexpr int SIMT_SMS = 148;

// Finds the (expert, first row, valid rows) of row tile `tile` when every expert's rows are tiled separately by `tm`: one
// warp, 32 experts at a time.  Returns false when `tile` is past the end.
__device__ bool locate_tile(const int* __restrict__ offset, int e_begin, int e_end, int tm, int tile, int& expert,
                            int& row0, int& rows) {
    const int lane = threadIdx.x & 31;
    int seen = 0;
    for (int e0 = e_begin; e0 < e_end; e0 += 32) {
        const int e = e0 + lane;
        const int beg = e < e_end ? offset[e] : 0, cnt = e < e_end ? offset[e + 1] - beg : 0;
        const int nt = (cnt + tm - 1) / tm;
        int incl = nt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += n;
        }
        const int first = seen + incl - nt;
        const unsigned hit = __ballot_sync(0xffffffffu, tile >= first && tile < first + nt);
        if (hit) {
            const int src = __ffs(hit) - 1;
            const int skip = (tile - __shfl_sync(0xffffffffu, first, src)) * tm;
            expert = e0 + src;
            row0 = __shfl_sync(0xffffffffu, beg, src) + skip;
            rows = min(tm, __shfl_sync(0xffffffffu, cnt, src) - skip);
            return true;
        }
        seen += __shfl_sync(0xffffffffu, incl, 31);
    }
    return false;
}

// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// Where the outputs go: g (DUAL), or row j to row out_pos[j] (or j) of `out`, or to the address out_row_ptr[out_pos[j]]; the
// residual is the same row of `resid`; mix_score != NULL applies the base_layer output mix.  With the combine step in here no
// routed copy of x and no result in expert order are written and read back: 300 tokens, 6 experts, 510 x 1022 one kernel of
// 3.6 us less.
struct SimtOutput {
    float* out;
    const float* resid;
    const int* out_pos;
    const float* mix_score;
    const unsigned long long* out_row_ptr;
};

// DUAL = true : out[j][n] = gelu(A W0^T) * (A W1^T), padded rows of N outputs   (N = d_ff, K = d_model)
// DUAL = false: out[.][n] = resid[.][n] + A W0^T, dense rows                    (N = d_model, K = d_ff)
// The k blocks are cut into `parts` shares whose sums are added in ascending k.  A tile (row tile, output tile; row tile major)
// belongs to a cluster of `parts` CTAs with a share each, or (WHOLE) to one CTA that takes the shares one after the other.
template <bool DUAL, int RI, bool WHOLE>
__global__ void __launch_bounds__(SIMT_THREADS, WHOLE && RI > 1 ? (DUAL ? 5 : 7) : 6)
ffn_simt_kernel(const int* __restrict__ offset, int e_begin, int e_end, int N, int K, int parts, const float* __restrict__ act,
                const float* __restrict__ w, const int* __restrict__ slot_of_expert, const SimtOutput o) {
    cg::cluster_group cluster = cg::this_cluster();
    const int S = WHOLE ? 1 : (int)cluster.num_blocks(), part = WHOLE ? 0 : (int)cluster.block_rank();
    const unsigned n_tiles = (unsigned)(N + TN - 1) / TN, tile = blockIdx.x / (unsigned)S;
    constexpr int TM = 16 * RI, WROWS = DUAL ? 2 * TN : TN, NB = DUAL ? 2 : 1;
    constexpr int BUF = (TM + WROWS) * PITCH;                 // floats of one buffer: token rows, then weight rows
    __shared__ __align__(16) float smem[2 * BUF];
    __shared__ int s_row[DUAL ? 1 : TM];                      // output rows of the tile, their addresses and mix coefficients
    __shared__ float* s_dst[DUAL ? 1 : TM];
    __shared__ float s_alpha[DUAL ? 1 : TM];
    __shared__ int s_info[4];
    if (threadIdx.x < 32) {
        int e = 0, r0 = 0, rows = 0;
        const bool ok = locate_tile(offset, e_begin, e_end, TM, (int)(tile / n_tiles), e, r0, rows);
        if (threadIdx.x == 0) {
            s_info[0] = ok ? 1 : 0;
            s_info[1] = e;
            s_info[2] = r0;
            s_info[3] = rows;
        }
    }
    __syncthreads();
    if (!s_info[0]) return;      // the same in every CTA of the cluster
    const int expert = s_info[1], row0 = s_info[2], rows = s_info[3];
    const int slot = slot_of_expert ? slot_of_expert[expert] : expert;
    const int n0 = (int)(tile % n_tiles) * TN, m0 = NB * n0;    // first output, first weight row (inside one 128-row block)
    const int KB = (K + TK - 1) / TK, MB = (NB * N + 127) / 128;
    const float* wt = w + (size_t)slot * (size_t)MB * KB * 4096 + ((size_t)(m0 >> 7) * KB) * 4096 + (size_t)(m0 & 127) * TK;
    const float* at = act + (size_t)row0 * KB * TK;
    const auto As = [&](int buf, int r) { return smem + buf * BUF + r * PITCH; };
    const auto Ws = [&](int buf, int r) { return smem + buf * BUF + (TM + r) * PITCH; };

    auto fetch = [&](int kb, int buf) {
        for (int i = threadIdx.x; i < TM * 8; i += SIMT_THREADS) {
            const int r = i >> 3, c = (i & 7) * 4;
            const bool valid = r < rows;
            copy16(As(buf, r) + c, at + (size_t)(valid ? r : 0) * KB * TK + kb * TK + c, valid);
        }
        for (int i = threadIdx.x; i < WROWS * 8; i += SIMT_THREADS) {
            const int r = i >> 3, c = (i & 7) * 4;
            // wi_0 and wi_1 rows apart, so that neighbouring outputs are neighbouring rows
            copy16(Ws(buf, DUAL ? (r & 1) * TN + (r >> 1) : r) + c, wt + (size_t)kb * 4096 + r * TK + c, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // token rows ty + 16 i, outputs tx + 8 j
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    float acc[NB][RI][4] = {};
    const int kb0 = KB * part / S, kb_end = KB * (part + 1) / S;
    fetch(kb0, kb0 & 1);
    // Where the outputs go; with four rows and more per warp while the first blocks are on their way: done row by row at the end, it
    // was a chain of trips to memory.
    const auto look_up_rows = [&]() {
        if (DUAL || (int)threadIdx.x >= rows) return;
        const int j = row0 + (int)threadIdx.x, row = o.out_pos ? o.out_pos[j] : j;
        s_row[threadIdx.x] = row;
        s_dst[threadIdx.x] = o.out_row_ptr ? reinterpret_cast<float*>(o.out_row_ptr[row]) : o.out + (size_t)row * N;
        if (o.mix_score) s_alpha[threadIdx.x] = mix_alpha(o.mix_score[j]);
    };
    if (RI > 1) look_up_rows();
    const auto multiply_block = [&](int kb) {
        const int buf = kb & 1;
        if (kb + 1 < kb_end) {
            fetch(kb + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; k += 4) {
            float4 a[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(As(buf, ty + 16 * i) + k);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(Ws(buf, b * TN + tx + 8 * j) + k);
#pragma unroll
                    for (int i = 0; i < RI; ++i) {
                        float s = acc[b][i][j];
                        s = fmaf(a[i].x, v.x, s);
                        s = fmaf(a[i].y, v.y, s);
                        s = fmaf(a[i].z, v.z, s);
                        acc[b][i][j] = fmaf(a[i].w, v.w, s);
                    }
                }
        }
        __syncthreads();    // the next round's fetch refills this buffer
    };
    if constexpr (!WHOLE) {
        for (int kb = kb0; kb < kb_end; ++kb) multiply_block(kb);
    } else {
        float total[NB][RI][4] = {};
        for (int kb = 0, share = 0; share < parts; ++share) {
            for (const int share_end = KB * (share + 1) / parts; kb < share_end; ++kb) multiply_block(kb);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        total[b][i][j] += acc[b][i][j];
                        acc[b][i][j] = share + 1 < parts ? 0.f : total[b][i][j];
                    }
        }
    }
    if constexpr (WHOLE && DUAL) {
#pragma unroll
        for (int i = 0; i < RI; ++i)
            if (ty + 16 * i < rows)
#pragma unroll
                for (int j = 0; j < 4; ++j)     // outputs past N are products of zero weights: the zeros the next GEMM's padding needs
                    o.out[(size_t)(row0 + ty + 16 * i) * padded_row(N) + n0 + tx + 8 * j] = gelu_dot(acc[0][i][j], acc[NB - 1][i][j]);
        return;
    }
    // Sums of the cluster's CTAs, added in ascending k; the CTAs share the outputs out.  A warp takes 32 consecutive outputs of a
    // row, so that what it stores is one run (the rows may lie in host memory), and several rows at a time: the stores may alias
    // the loads as far as the compiler knows, and one row after the other each would cost a trip to memory.
    constexpr int RED = TN + 8;                 // floats per row: the four rows a warp stores to end in different banks
    constexpr int AHEAD = WHOLE ? 4 : RI;
    static_assert(NB * TM * RED <= 2 * BUF, "the partial sums reuse the buffers");
    float* const red = smem;                    // [NB][TM][RED]
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) red[(b * TM + ty + 16 * i) * RED + tx + 8 * j] = acc[b][i][j];
    if (RI == 1) look_up_rows();
    if (WHOLE) __syncthreads();
    else cluster.sync();
    constexpr int WARPS = SIMT_THREADS / 32;
    const int lane = threadIdx.x & 31, n = n0 + lane, r_end = min(rows, TM * (part + 1) / S);
    for (int r0 = TM * part / S + (int)(threadIdx.x >> 5); r0 < r_end; r0 += WARPS * AHEAD) {
        float sum[AHEAD][NB] = {}, x[AHEAD];
        if (!DUAL)
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int r = r0 + WARPS * i;
                x[i] = r < r_end && n < N ? o.resid[(size_t)s_row[r] * N + n] : 0.f;
            }
        for (int q = 0; q < S; ++q) {
            const float* from = WHOLE ? red : cluster.map_shared_rank(red, q);
#pragma unroll
            for (int i = 0; i < AHEAD; ++i)
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    sum[i][b] += from[(b * TM + r0 + WARPS * i) * RED + lane];      // past `rows` too: never stored
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int r = r0 + WARPS * i;
            if (r >= r_end) continue;
            if (DUAL) {     // outputs past N are products of zero weights: the zeros the next GEMM's padding needs
                o.out[(size_t)(row0 + r) * padded_row(N) + n] = gelu_dot(sum[i][0], sum[i][NB - 1]);
            } else if (n < N) {
                float y = x[i] + sum[i][0];
                if (o.mix_score) y = mix_value(s_alpha[r], 1.0f - s_alpha[r], y, x[i]);
                s_dst[r][n] = y;
            }
        }
    }
    if (!WHOLE) cluster.sync();      // nobody leaves while its sums are being read
}

}  // namespace

// Grouped FFN over experts [e_begin, e_end); T rows in expert-contiguous order.
//   h [T][padded_row(D)], g [T][padded_row(F)] (scratch); output as in FfnUmma
//   slot_of_expert (device, may be NULL = identity) maps expert -> weight slot.
int launch_ffn_simt(long long T, int D, int F, int e_begin, int e_end, const int* offset, const int* slot_of_expert,
                    const float* h, const float* w01, const float* wo, float* g, const float* resid, float* out,
                    const int* out_pos, const float* mix_score, const unsigned long long* out_row_ptr, cudaStream_t stream) {
    if (T == 0 || e_begin >= e_end) return INFMOE_OK;
    const int experts = e_end - e_begin;
    // 16-row tiles when an expert has about that many rows at most: a 64-row tile would multiply zeros
    const bool few = T <= 16ll * experts;
    const int tm = few ? 16 : 64;
    const unsigned row_tiles = (unsigned)((T + tm - 1) / tm + experts);
    // Not chained (launch_chained): blocks put on the SMs while those of the kernel before are still there crowd on the
    // idle ones, and there are only a few per SM.  The pass of 300 tokens took 195 us so, 126 with a late trigger.
    const auto launch = [&](auto dual, int N, int K, const float* act, const float* w, const SimtOutput& o) {
        constexpr bool DUAL = decltype(dual)::value;
        // shares of K: by K alone, so that a row's additions do not depend on the other rows of the call
        const unsigned parts = K > 7 * TK ? 4 : K > 3 * TK ? 2 : 1, tiles = (unsigned)((N + TN - 1) / TN) * row_tiles;
        // One CTA per tile where there is nothing to share, and where the tiles alone keep the SMs busy: a cluster pays for its start,
        // its sums and barriers with every share.  Tiles: half of one per expert may be missing from its last.  The line in tiles per
        // SM; us of the kernel, cluster | one CTA per tile, tiles (experts x d_model x d_ff, tokens):
        //   first GEMM      6 x 510 x 1022: 576: 77 | 80, 832: 110 | 104, 2240: 267 | 233, 8288: 994 | 846; 4 x 2050 x 4098: 645: 251 | 313
        //   second GEMM     half the work per tile: 1072 (4096 tokens) 144 | 159, 64 x 510 x 1022 1504: 189 | 179, 6 x 510 x 1022 4144: 529 | 494
        //   16-row tiles    either GEMM: 4 x 2050 x 4098 774: 243 | 254, 64 x 510 x 1022 1152: 104 | 97, 1536: 121 | 115
        //   64-row tiles, shares of three k blocks and less    4 x 130 x 258: 117: 11.8 | 12.4, 234: 18.1 | 14.7, 594: 35 | 30
        // Passes, before the clusters, with clusters always, now: 6 x 510 x 1022, 4096 tokens 403, 446, 401, 16384 1379, 1631, 1408;
        // 4 x 130 x 258, 4096 69.5, 80.4, 69.2; 4 x 66 x 130, 300 23.8, 28.0, 22.4; 4 x 2050 x 4098, 1000 1414, 1493, 1376.
        const long long busy = (long long)((N + TN - 1) / TN) * (T / tm + (experts < T ? experts : T) / 2);
        const bool short_shares = !few && (K + TK - 1) / TK <= 3 * (int)parts;
        const bool whole = parts == 1 || busy >= SIMT_SMS * (short_shares ? 1 : few ? 6 : DUAL ? 5 : 10);
        const auto kern = few ? (whole ? ffn_simt_kernel<DUAL, 1, true> : ffn_simt_kernel<DUAL, 1, false>)
                              : (whole ? ffn_simt_kernel<DUAL, 4, true> : ffn_simt_kernel<DUAL, 4, false>);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(whole ? tiles : tiles * parts);
        cfg.blockDim = dim3(SIMT_THREADS);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = parts;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = whole ? 0 : 1;
        return cudaLaunchKernelEx(&cfg, kern, offset, e_begin, e_end, N, K, (int)parts, act, w, slot_of_expert, o);
    };
    INFMOE_CUDA_TRY(launch(std::true_type(), F, D, h, w01, SimtOutput{g, nullptr, nullptr, nullptr, nullptr}));
    INFMOE_CUDA_TRY(launch(std::false_type(), D, F, (const float*)g, wo,
                           SimtOutput{out, resid, out_pos, mix_score, out_row_ptr}));
    note_launch(2);
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

}  // namespace infmoe
