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
// Bound by FP32 FMA issue for many rows per expert, by the number of CTAs for few.  A CTA computes 16 RI token rows x 32
// outputs; a thread RI x 4 (x 2 when both matrices are multiplied) of them.  K blocks of 32 are fetched by 16-byte
// cp.async into two buffers.  Both operands stay row-major in shared memory at a pitch of 36 floats, and a thread reads
// four k of a row at a time: 4 + 8 128-bit loads for 128 multiply-adds, without bank conflicts (the eight weight rows a
// warp reads at once start 4 banks apart; token rows are broadcasts).  Every output is one chain of FMAs in ascending k.
// Layer of 300 tokens, 6 experts, 510 x 1022: 423 -> 103 us (it was 64 x 64 tiles of scalar loads, one buffer, TF32 head
// and tail planes added on the fly).
#include "common.cuh"
#include "kernels.h"

namespace infmoe {

namespace {

constexpr int SIMT_THREADS = 128;
constexpr int TN = 32;       // outputs per CTA
constexpr int TK = 32;       // one k block of the weight tiles
constexpr int PITCH = TK + 4;

// Finds the (expert, first row, valid rows) of row tile `tile` when every expert's rows are tiled separately by `tm`.
// Returns false when `tile` is past the end.
__device__ bool locate_tile(const int* __restrict__ offset, int e_begin, int e_end, int tm, int tile, int& expert,
                            int& row0, int& rows) {
    int seen = 0;
    for (int e = e_begin; e < e_end; ++e) {
        const int beg = offset[e], cnt = offset[e + 1] - beg;
        const int nt = (cnt + tm - 1) / tm;
        if (tile < seen + nt) {
            expert = e;
            row0 = beg + (tile - seen) * tm;
            rows = min(tm, beg + cnt - row0);
            return true;
        }
        seen += nt;
    }
    return false;
}

// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// DUAL = true : out[j][n] = gelu(A W0^T) * (A W1^T), padded rows of N outputs   (N = d_ff, K = d_model)
// DUAL = false: out[j][n] = resid[j][n] + A W0^T, dense rows                    (N = d_model, K = d_ff)
template <bool DUAL, int RI>
__global__ void __launch_bounds__(SIMT_THREADS)
ffn_simt_kernel(const int* __restrict__ offset, int e_begin, int e_end, int N, int K, const float* __restrict__ act,
                const float* __restrict__ w, const int* __restrict__ slot_of_expert, const float* __restrict__ resid,
                float* __restrict__ out) {
    const unsigned n_tiles = (unsigned)(N + TN - 1) / TN;     // grid: row tile major
    constexpr int TM = 16 * RI, WROWS = DUAL ? 2 * TN : TN, NB = DUAL ? 2 : 1;
    __shared__ __align__(16) float As[2][TM][PITCH];
    __shared__ __align__(16) float Ws[2][WROWS][PITCH];
    __shared__ int s_info[4];
    if (threadIdx.x == 0) {
        int e = 0, r0 = 0, rows = 0;
        const bool ok = locate_tile(offset, e_begin, e_end, TM, blockIdx.x / n_tiles, e, r0, rows);
        s_info[0] = ok ? 1 : 0;
        s_info[1] = e;
        s_info[2] = r0;
        s_info[3] = rows;
    }
    __syncthreads();
    if (!s_info[0]) return;
    const int expert = s_info[1], row0 = s_info[2], rows = s_info[3];
    const int slot = slot_of_expert ? slot_of_expert[expert] : expert;
    const int n0 = (int)(blockIdx.x % n_tiles) * TN, m0 = NB * n0;    // first output, first weight row (inside one 128-row block)
    const int KB = (K + TK - 1) / TK, MB = (NB * N + 127) / 128;
    const float* wt = w + (size_t)slot * (size_t)MB * KB * 4096 + ((size_t)(m0 >> 7) * KB) * 4096 + (size_t)(m0 & 127) * TK;
    const float* at = act + (size_t)row0 * KB * TK;

    auto fetch = [&](int kb, int buf) {
        for (int i = threadIdx.x; i < TM * 8; i += SIMT_THREADS) {
            const int r = i >> 3, c = (i & 7) * 4;
            const bool valid = r < rows;
            copy16(&As[buf][r][c], at + (size_t)(valid ? r : 0) * KB * TK + kb * TK + c, valid);
        }
        for (int i = threadIdx.x; i < WROWS * 8; i += SIMT_THREADS) {
            const int r = i >> 3, c = (i & 7) * 4;
            // wi_0 and wi_1 rows apart, so that neighbouring outputs are neighbouring rows
            copy16(&Ws[buf][DUAL ? (r & 1) * TN + (r >> 1) : r][c], wt + (size_t)kb * 4096 + r * TK + c, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // token rows ty + 16 i, outputs tx + 8 j
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    float acc[NB][RI][4] = {};
    fetch(0, 0);
    for (int kb = 0; kb < KB; ++kb) {
        const int buf = kb & 1;
        if (kb + 1 < KB) {
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
            for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(&As[buf][ty + 16 * i][k]);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(&Ws[buf][b * TN + tx + 8 * j][k]);
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
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int r = ty + 16 * i;
        if (r >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 8 * j;
            if (DUAL) {     // outputs past N are products of zero weights: the zeros the next GEMM's padding needs
                out[(size_t)(row0 + r) * padded_row(N) + n] = gelu_dot(acc[0][i][j], acc[NB - 1][i][j]);
            } else if (n < N) {
                const size_t o = (size_t)(row0 + r) * N + n;
                out[o] = resid[o] + acc[0][i][j];
            }
        }
    }
}

}  // namespace

// Grouped FFN over experts [e_begin, e_end); T rows in expert-contiguous order.
//   h [T][padded_row(D)], g [T][padded_row(F)] (scratch), routed [T][D], post [T][D]
//   slot_of_expert (device, may be NULL = identity) maps expert -> weight slot.
int launch_ffn_simt(long long T, int D, int F, int e_begin, int e_end, const int* offset, const int* slot_of_expert,
                    const float* h, const float* w01, const float* wo, const float* routed, float* g, float* post,
                    cudaStream_t stream) {
    if (T == 0 || e_begin >= e_end) return INFMOE_OK;
    const int experts = e_end - e_begin;
    // 16-row tiles when an expert has about that many rows at most: a 64-row tile would multiply zeros
    const bool few = T <= 16ll * experts;
    const int tm = few ? 16 : 64;
    const unsigned row_tiles = (unsigned)((T + tm - 1) / tm + experts);
    const unsigned g1 = (unsigned)((F + TN - 1) / TN) * row_tiles, g2 = (unsigned)((D + TN - 1) / TN) * row_tiles;
    auto k1 = few ? ffn_simt_kernel<true, 1> : ffn_simt_kernel<true, 4>;
    auto k2 = few ? ffn_simt_kernel<false, 1> : ffn_simt_kernel<false, 4>;
    // Not chained (launch_chained): blocks put on the SMs while those of the kernel before are still there crowd on the
    // idle ones, and there are only a few per SM.  The pass of 300 tokens took 195 us so, 126 with a late trigger.
    k1<<<g1, SIMT_THREADS, 0, stream>>>(offset, e_begin, e_end, F, D, h, w01, slot_of_expert, nullptr, g);
    k2<<<g2, SIMT_THREADS, 0, stream>>>(offset, e_begin, e_end, D, F, g, wo, slot_of_expert, routed, post);
    note_launch(2);
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

}  // namespace infmoe
