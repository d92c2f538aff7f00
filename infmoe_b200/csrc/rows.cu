// Row-wise kernels of the MoE layer: scatter into expert-contiguous order,
// gather / mix back to token order, LayerNorm, gelu-dot and the splits that feed
// the GEMMs.  All of them are pure HBM streaming:
// one warp per row, 128-bit loads and stores, rows of one warp contiguous.
//
// Reference counterparts (all scalar 4-byte copies, one CTA of 256 threads per row):
//   batch_scatter_feature_and_weight_kernel  plugin/cuda/moe.cu:98-113
//   batch_gather_kernel                      plugin/cuda/moe.cu:89-96
//   fused_batch_mix_and_gather_kernel        plugin/cuda/moe.cu:115-127
//   cuApplyLayerNorm                         plugin/cuda/ops/layernorm.cu:136-174
//   gelu_dot functor via thrust::transform   plugin/cuda/ops/gelu.cu:6-25
#include <cooperative_groups.h>

#include <climits>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace infmoe {

namespace {

constexpr int ROW_WARPS = 8;

__device__ __forceinline__ void copy_row(const float* __restrict__ src, float* __restrict__ dst, int D, bool vec,
                                         int lane) {
    if (vec) {
        const float4* s4 = reinterpret_cast<const float4*>(src);
        float4* d4 = reinterpret_cast<float4*>(dst);
        for (int i = lane; i < D / 4; i += 32) d4[i] = s4[i];
    } else {
        for (int i = lane; i < D; i += 32) dst[i] = src[i];
    }
}

// routed[j,:] = X[pos[j],:]; rcoeff[j] = coeff[pos[j]]
__global__ void __launch_bounds__(ROW_WARPS * 32)
scatter_kernel(long long T, int D, int vec, const float* X, const float* coeff,
               const int* pos, float* __restrict__ routed, float* __restrict__ rcoeff) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= T) return;
    const int p = pos[j];
    copy_row(X + (long long)p * D, routed + j * D, D, vec != 0, lane);
    if (lane == 0 && coeff && rcoeff) rcoeff[j] = coeff[p];
}

// The layer's fused scatter: X[pos[j],:] -> its per-expert LayerNorm h = LN(x; gamma_e) (T5FFLayer.cc:99-103), ready
// for the grouped GEMM.  The expert of row j is gate[pos[j]].  Rows at or past *valid_rows (tokens without an expert,
// empty receive slots) are skipped.
//
// For the CUDA-core GEMM: the routed score, and h in FP32, rows padded with zeros to whole groups of 32.
__device__ __forceinline__ void warp_ln_rows(const float* __restrict__ src, const float* __restrict__ gamma, int D,
                                             bool vec, float* __restrict__ h) {
    const int lane = threadIdx.x & 31;
    float mean, rstd;
    warp_row_stats(src, D, vec, mean, rstd);
    for (int base = 4 * lane; base < (int)padded_row(D); base += 128) {
        float hh[4] = {0.f, 0.f, 0.f, 0.f};
        if (base < D) {
            const float4 v = load_row4(src, base, D, vec), g = load_row4(gamma, base, D, vec);
            const float vv[4] = {v.x, v.y, v.z, v.w}, gg[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (base + k < D) hh[k] = ln_apply(vv[k], mean, rstd, gg[k]);
        }
        *reinterpret_cast<float4*>(h + base) = make_float4(hh[0], hh[1], hh[2], hh[3]);
    }
}

__global__ void __launch_bounds__(ROW_WARPS * 32)
scatter_ln_rows_kernel(long long T, int D, int vec, const float* X, const float* score,
                       const int* pos, const int* gate, const float* gamma_all,
                       const int* valid_rows, float* __restrict__ rscore, float* __restrict__ h) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= T || (valid_rows && j >= *valid_rows)) return;
    const int p = pos[j];
    warp_ln_rows(X + (long long)p * D, gamma_all + (long long)gate[p] * D, D, vec != 0, h + j * (long long)padded_row(D));
    if (lane == 0 && rscore && score) rscore[j] = score[p];
}

// One warp: h = LN(src; gamma) as FP16 pairs scaled by a power of two of the row, and the row's two numbers.
__device__ __forceinline__ void warp_ln_pack(const float* __restrict__ src, const float* __restrict__ gamma, int D,
                                             bool vec, uint16_t* __restrict__ pack_row, float2* __restrict__ info) {
    const int lane = threadIdx.x & 31;
    float mean, rstd;
    warp_row_stats(src, D, vec, mean, rstd);
    auto load_h = [&](int base, float (&h)[4]) {
        const float4 v = load_row4(src, base, D, vec), g = load_row4(gamma, base, D, vec);
        const float vv[4] = {v.x, v.y, v.z, v.w}, gg[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = base + k < D ? ln_apply(vv[k], mean, rstd, gg[k]) : 0.f;
    };
    float top = 0.f;
    for (int base = 4 * lane; base < D; base += 128) {
        float h[4];
        load_h(base, h);
#pragma unroll
        for (int k = 0; k < 4; ++k) top = fmaxf(top, fabsf(h[k]));
    }
    const int s = row_exponent(warp_max(top));
    const float scale = exp2_int(s);
    float squares = 0.f;
    for (int base = 4 * lane; base < ((D + 31) & ~31); base += 128) {
        float h[4] = {0.f, 0.f, 0.f, 0.f};
        if (base < D) load_h(base, h);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            h[k] = __fmul_rn(h[k], scale);
            squares = fmaf(h[k], h[k], squares);
        }
        store_pack4(pack_row, base, h);
    }
    squares = warp_xor_sum(squares);
    if (lane == 0) *info = token_row_info(s, squares);
}

// The scatter for the tensor-core GEMM, of rows j0 .. j0 + T - 1.  The LayerNorm weights are gamma' (see SplitExpert), which
// lies with the experts' planes.
struct ExpertGamma {
    const float* base;              // first expert
    size_t stride;                  // floats from one expert to the next
    __device__ __forceinline__ const float* of(int e) const { return base + stride * (size_t)e; }
};
__global__ void __launch_bounds__(ROW_WARPS * 32)
scatter_ln_pack_kernel(long long j0, long long T, int D, int vec, const float* X,
                       const float* score, const int* pos, const int* gate,
                       const ExpertGamma gamma, const int* valid_rows, float* __restrict__ rscore,
                       uint16_t* __restrict__ h, float2* __restrict__ row_info) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const long long j = j0 + (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= j0 + T || (valid_rows && j >= *valid_rows)) return;
    const int p = pos[j];
    warp_ln_pack(X + (long long)p * D, gamma.of(gate[p]), D, vec != 0,
                 h + j * (long long)pack_pitch(D), row_info + j);
    if (lane == 0 && rscore && score) rscore[j] = score[p];
}

// The same for aligned rows of up to 128 * NV floats, with more bytes in flight per warp: the whole row is
// fetched into registers by back-to-back 128-bit loads (NV per lane) before any of it is used, so it crosses HBM
// once in one burst and the statistics passes and the split run from registers.  The additions of the LayerNorm happen
// in the order of warp_row_stats, so h has the same bits.  Few rows per SM (4096 rows on 148 SMs) would
// otherwise leave the memory system half idle.  The expert's LayerNorm weights are fetched into shared memory by
// cp.async while the row is on its way, so the output loop never waits for L2.
// Bound by HBM: reads 4 D and writes 4 D bytes per row (a third less than the two planes it wrote before).
template <int NV>
struct RowInRegisters {
    float4 v[NV];
    float mean, rstd;
    static __device__ __forceinline__ int lane() { return threadIdx.x & 31; }
    __device__ __forceinline__ void fetch(const float* __restrict__ row, int D) {
        const float4* src = reinterpret_cast<const float4*>(row);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int base = 4 * lane() + 128 * i;
            v[i] = base < D ? src[base >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    // LayerNorm weights to shared memory; every lane reads back only what it fetched itself (ln_pack waits for it)
    static __device__ __forceinline__ void fetch_gamma(float4* s_gamma, const float* __restrict__ gamma, int D) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int base = 4 * lane() + 128 * i;
            if (base < D) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_gamma + (base >> 2));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(gamma + base) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void stats(int D) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (4 * lane() + 128 * i < D) s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v[i].x), v[i].y), v[i].z), v[i].w);
        mean = __fdiv_rn(warp_xor_sum(s), (float)D);
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (4 * lane() + 128 * i < D) {
                float d = __fsub_rn(v[i].x, mean);
                q = __fmaf_rn(d, d, q);
                d = __fsub_rn(v[i].y, mean);
                q = __fmaf_rn(d, d, q);
                d = __fsub_rn(v[i].z, mean);
                q = __fmaf_rn(d, d, q);
                d = __fsub_rn(v[i].w, mean);
                q = __fmaf_rn(d, d, q);
            }
        const float var = __fdiv_rn(warp_xor_sum(q), (float)D);
        rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var, 1e-6f)));
    }
    __device__ __forceinline__ void ln_pack(const float4* s_gamma, int D, uint16_t* __restrict__ pack_row, float2* info) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        float top = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int base = 4 * lane() + 128 * i;
            if (base >= D) continue;
            const float4 g = s_gamma[base >> 2];
            v[i].x = ln_apply(v[i].x, mean, rstd, g.x);
            v[i].y = ln_apply(v[i].y, mean, rstd, g.y);
            v[i].z = ln_apply(v[i].z, mean, rstd, g.z);
            v[i].w = ln_apply(v[i].w, mean, rstd, g.w);
            top = fmaxf(fmaxf(fmaxf(top, fabsf(v[i].x)), fmaxf(fabsf(v[i].y), fabsf(v[i].z))), fabsf(v[i].w));
        }
        const int exponent = row_exponent(warp_max(top));
        const float scale = exp2_int(exponent);
        const int k_end = (D + 31) & ~31;
        float squares = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int base = 4 * lane() + 128 * i;
            if (base >= k_end) continue;
            const float x[4] = {__fmul_rn(v[i].x, scale), __fmul_rn(v[i].y, scale), __fmul_rn(v[i].z, scale),
                                __fmul_rn(v[i].w, scale)};     // zeros past the row
#pragma unroll
            for (int k = 0; k < 4; ++k) squares = fmaf(x[k], x[k], squares);
            store_pack4(pack_row, base, x);
        }
        squares = warp_xor_sum(squares);
        if (lane() == 0) *info = token_row_info(exponent, squares);
    }
};

template <int NV>
__global__ void __launch_bounds__(128)
scatter_ln_pack_reg_kernel(long long j0, long long T, int D, const float* X,
                           const float* score, const int* pos, const int* gate,
                           const ExpertGamma expert_gamma, const int* valid_rows, float* __restrict__ rscore,
                           uint16_t* __restrict__ h, float2* __restrict__ row_info) {
    pdl_wait();
    pdl_trigger();
    const long long j = j0 + (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (j >= j0 + T || (valid_rows && j >= *valid_rows)) return;
    extern __shared__ __align__(16) float4 s_gamma_all[];     // [4 warps][NV * 32]
    float4* s_gamma = s_gamma_all + (threadIdx.x >> 5) * (NV * 32);
    const int p = pos[j];
    const int e = gate[p];
    RowInRegisters<NV> row;
    row.fetch(X + (long long)p * D, D);
    row.fetch_gamma(s_gamma, expert_gamma.of(e), D);
    row.stats(D);
    row.ln_pack(s_gamma, D, h + j * (long long)pack_pitch(D), row_info + j);
    if ((threadIdx.x & 31) == 0 && rscore && score) rscore[j] = score[p];
}

// f(t, gate[t]) for t = threadIdx.x, + THREADS, ... below T, with eight loads on their way together (one by one they are a trip
// to L2 each, 0.7 us, sixteen of them for a block that looks at 4096 gates).
template <int THREADS, typename F>
__device__ __forceinline__ void for_gates(const int* __restrict__ gate, int T, const F& f) {
    for (int t0 = threadIdx.x; t0 < T; t0 += 8 * THREADS) {
        int g[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) g[i] = t0 + i * THREADS < T ? gate[t0 + i * THREADS] : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (t0 + i * THREADS < T) f(t0 + i * THREADS, g[i]);
    }
}

// count[] and offset[] of the T gates by one block of THREADS threads, and zero[] cleared on the way.
template <int THREADS>
__device__ __forceinline__ void histogram_block(int* hist, int T, int E, const int* __restrict__ gate, int* __restrict__ count,
                                                int* __restrict__ offset, int* __restrict__ status, int* __restrict__ zero,
                                                int zero_count) {
    const int tid = threadIdx.x, lane = tid & 31;
    for (int e = tid; e <= E; e += THREADS) hist[e] = 0;
    for (int i = tid; i < zero_count; i += THREADS) zero[i] = 0;
    __syncthreads();
    bool bad = false;
    for_gates<THREADS>(gate, T, [&](int, int e) {
        const bool ok = e >= 0 && e < E;
        bad |= !ok;
        atomicAdd(&hist[ok ? e : E], 1);
    });
    if (bad && status) atomicOr(status, STATUS_BAD_GATE);
    __syncthreads();
    if (tid < 32) {
        int carry = 0;
        for (int e0 = 0; e0 <= E; e0 += 32) {     // exclusive scan, 32 buckets at a time
            const int e = e0 + lane, c = e <= E ? hist[e] : 0;
            int incl = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += n;
            }
            if (e <= E) offset[e] = carry + incl - c;     // offset[E]: tokens that have an expert
            if (e < E) count[e] = c;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

// Few tokens: dispatch metadata (dispatch.cu) and the scatter in one launch.  A block per token counts the tokens that
// come before its own (smaller expert, or same expert and smaller index) while its row and the expert's LayerNorm weight
// are on their way to shared memory, so nothing waits for a separate kernel of one cluster and then for pos[] and
// gate[]; one more block writes count[] and offset[].  T blocks read T gates each, from L2: 4 MB for 1024 tokens, the
// most it takes.  Results, LayerNorm bits included, are those of dispatch_kernel and the scatter kernels.
// Layer of 32 tokens, 4 experts, 64 x 256: 36 -> 24 us together with launch_chained; 1 token, 32 experts, 4096 x 10240:
// 149 -> 136.
// early: the kernel before is the routing, whose blocks start their successor only after their own wait.  So all that was
// enqueued before the routing is complete, the tokens are there, and a block fetches its row and computes the row's
// statistics while the routing is still running.
constexpr int DS_THREADS = 128;
template <bool PACK>
__global__ void __launch_bounds__(DS_THREADS)
dispatch_scatter_kernel(int T, int D, int E, int vec, const float* X, const float* score,
                        const int* gate, const ExpertGamma expert_gamma, int* __restrict__ pos,
                        int* __restrict__ count, int* __restrict__ offset, int* __restrict__ status,
                        int* __restrict__ zero, int zero_count, float* __restrict__ rscore, void* __restrict__ h,
                        float2* __restrict__ row_info, int early) {
    extern __shared__ __align__(16) float ds_smem[];
    __shared__ int s_before[DS_THREADS / 32];
    __shared__ float s_top[DS_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!early || (int)blockIdx.x == T) {
        pdl_wait();
        pdl_trigger();
    }
    if ((int)blockIdx.x == T) {
        histogram_block<DS_THREADS>(reinterpret_cast<int*>(ds_smem), T, E, gate, count, offset, status, zero, zero_count);
        return;
    }
    const int t = (int)blockIdx.x;
    const int P = (int)padded_row(D);
    float *s_x = ds_smem, *s_g = ds_smem + P;
    const auto fetch = [&](float* dst, const float* src) {
        if (vec) {
            for (int k = 4 * tid; k < D; k += 4 * DS_THREADS) {
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + k);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + k) : "memory");
            }
        } else {
#pragma unroll 4
            for (int k = tid; k < D; k += DS_THREADS) dst[k] = src[k];
        }
        for (int k = D + tid; k < P; k += DS_THREADS) dst[k] = 0.f;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(s_x, X + (size_t)t * D);
    float mean, rstd;
    const auto stats = [&]() { warp_row_stats(s_x, D, (D & 3) == 0, mean, rstd); };     // every warp for itself
    if (early) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        stats();
        pdl_wait();
        pdl_trigger();
    }
    int e = gate[t];
    if (e < 0 || e >= E) e = E;
    fetch(s_g, expert_gamma.of(e < E ? e : 0));
    int before = 0;
    for (int o = tid; o < T; o += DS_THREADS) {
        int g = gate[o];
        if (g < 0 || g >= E) g = E;
        before += (g < e || (g == e && o < t)) ? 1 : 0;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_before[warp] = before;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int j = 0;
#pragma unroll
    for (int w = 0; w < DS_THREADS / 32; ++w) j += s_before[w];
    if (tid == 0) {
        pos[j] = t;
        if (e < E && rscore && score) rscore[j] = score[t];
    }
    if (e == E) return;              // no expert: nobody reads the row
    if (!early) {
        stats();
        __syncthreads();
    }
    float top = 0.f;
    for (int k = 4 * tid; k < P; k += 4 * DS_THREADS) {
        float* x = s_x + k;
        const float4 g = *reinterpret_cast<const float4*>(s_g + k);
        float4 v = *reinterpret_cast<const float4*>(x);
        v.x = k < D ? ln_apply(v.x, mean, rstd, g.x) : 0.f;
        v.y = k + 1 < D ? ln_apply(v.y, mean, rstd, g.y) : 0.f;
        v.z = k + 2 < D ? ln_apply(v.z, mean, rstd, g.z) : 0.f;
        v.w = k + 3 < D ? ln_apply(v.w, mean, rstd, g.w) : 0.f;
        if (PACK) {
            top = fmaxf(fmaxf(fmaxf(top, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
            *reinterpret_cast<float4*>(x) = v;            // the thread's own values again below
        } else {
            *reinterpret_cast<float4*>(static_cast<float*>(h) + (size_t)j * P + k) = v;
        }
    }
    if (!PACK) return;
    top = warp_max(top);
    if (lane == 0) s_top[warp] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < DS_THREADS / 32; ++w) top = fmaxf(top, s_top[w]);
    const int s = row_exponent(top);
    const float scale = exp2_int(s);
    uint16_t* pack_row = static_cast<uint16_t*>(h) + (size_t)j * pack_pitch(D);
    for (int k = 4 * tid; k < P; k += 4 * DS_THREADS) {
        float4 v = *reinterpret_cast<const float4*>(s_x + k);
        v = make_float4(__fmul_rn(v.x, scale), __fmul_rn(v.y, scale), __fmul_rn(v.z, scale), __fmul_rn(v.w, scale));
        *reinterpret_cast<float4*>(s_x + k) = v;
        const float x[4] = {v.x, v.y, v.z, v.w};
        store_pack4(pack_row, k, x);
    }
    __syncthreads();
    if (warp == 0) {                 // the sum of squares in the order of the other scatter kernels
        float squares = 0.f;
        for (int k = 4 * lane; k < P; k += 128) {
            const float4 v = *reinterpret_cast<const float4*>(s_x + k);
            squares = fmaf(v.x, v.x, squares);
            squares = fmaf(v.y, v.y, squares);
            squares = fmaf(v.z, v.z, squares);
            squares = fmaf(v.w, v.w, squares);
        }
        squares = warp_xor_sum(squares);
        if (lane == 0) row_info[j] = token_row_info(s, squares);
    }
}

// The same for more tokens, aligned rows of up to 128 NV floats: eight tokens per block, a warp and its registers for each.
// The blocks read T / 8 x T gates, from L2, and compare each with eight: key (gate, token) below the own one.  4096
// tokens are the most it takes: 8 MB and about 1.5 us of comparisons, against a kernel of one cluster between routing and
// scatter.  Bound by latency: the gates' trips to L2, then the LayerNorm weights', in one to two rounds of blocks (three or four
// to an SM by registers).  Dispatch and scatter, us, each timed by itself: 4096 tokens of 512 floats 12 + 10 -> 14.7, 1024 floats 11
// + 12 -> 16.8, 2500 tokens of 512 floats 11 + 10 -> 10.9, 2048 tokens of 1028 floats 12.6 + 10.5 -> 12.3 (64 experts), 4096 of 2048
// 11.1 + 20.4 -> 22.9.  The line at 4096 is where the measurements end, not where the two forms meet: the comparisons grow with
// T squared, and at the line this one is still ahead.  Whole passes, 5 experts, d_ff 64, at 4096 | 4097 tokens: 256 floats 33.1 |
// 36.5, 1024 57.2 | 58.2, 2048 98.6 | 101.8.
constexpr int DM_THREADS = 256;
constexpr int DM_TOKENS = DM_THREADS / 32;
constexpr int DM_MAX_TOKENS = 4096;
template <int NV>
__global__ void __launch_bounds__(DM_THREADS, NV <= 4 ? 4 : NV <= 8 ? 3 : 2)
dispatch_scatter_reg_kernel(int T, int D, int E, const float* X, const float* score,
                            const int* gate, const ExpertGamma expert_gamma, int* __restrict__ pos,
                            int* __restrict__ count, int* __restrict__ offset, int* __restrict__ status,
                            int* __restrict__ zero, int zero_count, float* __restrict__ rscore, uint16_t* __restrict__ h,
                            float2* __restrict__ row_info, int early) {
    extern __shared__ __align__(16) float4 dm_gamma[];     // [warp][NV * 32]; histogram block: E + 1 words
    __shared__ int s_before[DM_TOKENS][DM_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = ((int)blockIdx.x - 1) * DM_TOKENS, t = t0 + warp;
    if (blockIdx.x == 0) {      // first, because it takes as long as any
        pdl_wait();
        pdl_trigger();
        histogram_block<DM_THREADS>(reinterpret_cast<int*>(dm_gamma), T, E, gate, count, offset, status, zero, zero_count);
        return;
    }
    RowInRegisters<NV> row;
    if (!early) pdl_wait();
    row.fetch(X + (size_t)min(t, T - 1) * D, D);
    row.stats(D);
    if (early) pdl_wait();
    pdl_trigger();
    const auto key_of = [&](int o, int g) { return (g >= 0 && g < E ? g : E) * DM_MAX_TOKENS + o; };
    const auto key = [&](int o) { return key_of(o, gate[o]); };
    const int own = key(min(t, T - 1)), e = own / DM_MAX_TOKENS;
    float4* const s_gamma = dm_gamma + warp * (NV * 32);
    row.fetch_gamma(s_gamma, expert_gamma.of(e < E ? e : 0), D);
    int keys[DM_TOKENS], before[DM_TOKENS] = {};
#pragma unroll
    for (int j = 0; j < DM_TOKENS; ++j) keys[j] = key(min(t0 + j, T - 1));
    for_gates<DM_THREADS>(gate, T, [&](int o, int g) {
        const int k = key_of(o, g);
#pragma unroll
        for (int j = 0; j < DM_TOKENS; ++j) before[j] += k < keys[j] ? 1 : 0;
    });
#pragma unroll
    for (int j = 0; j < DM_TOKENS; ++j) {
        const int n = __reduce_add_sync(0xffffffffu, before[j]);
        if (lane == 0) s_before[j][warp] = n;
    }
    __syncthreads();
    if (t >= T) return;
    int j = 0;
#pragma unroll
    for (int w = 0; w < DM_THREADS / 32; ++w) j += s_before[warp][w];
    if (lane == 0) {
        pos[j] = t;
        if (e < E && rscore && score) rscore[j] = score[t];
    }
    if (e == E) return;              // no expert: nobody reads the row
    row.ln_pack(s_gamma, D, h + (size_t)j * pack_pitch(D), row_info + j);
}

// out[pos[j],:] = in[j,:] for the rows below *valid_rows (all rows when valid_rows is NULL)
__global__ void __launch_bounds__(ROW_WARPS * 32)
gather_kernel(long long T, int D, int vec, const float* in, const int* pos,
              const int* valid_rows, float* __restrict__ out) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= T || (valid_rows && j >= *valid_rows)) return;
    copy_row(in + j * D, out + (long long)pos[j] * D, D, vec != 0, lane);
}

// alpha = 1 / (1 + exp(-coeff[j])); out[pos[j],:] = alpha * post[j,:] + (1 - alpha) * routed[j,:]
// (sigmoid: plugin/cuda/common.cuh:24-27)
__global__ void __launch_bounds__(ROW_WARPS * 32)
mix_gather_kernel(long long T, int D, int vec, const int* pos, const float* routed,
                  const float* post, const float* coeff,
                  const int* valid_rows, float* __restrict__ out) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= T || (valid_rows && j >= *valid_rows)) return;
    const float alpha = mix_alpha(coeff[j]);
    const float beta = 1.0f - alpha;
    const float* a = post + j * D;
    const float* b = routed + j * D;
    float* o = out + (long long)pos[j] * D;
    if (vec) {
        for (int i = lane; i < D / 4; i += 32) {
            const float4 x = reinterpret_cast<const float4*>(a)[i];
            const float4 y = reinterpret_cast<const float4*>(b)[i];
            float4 r;
            r.x = mix_value(alpha, beta, x.x, y.x);
            r.y = mix_value(alpha, beta, x.y, y.y);
            r.z = mix_value(alpha, beta, x.z, y.z);
            r.w = mix_value(alpha, beta, x.w, y.w);
            reinterpret_cast<float4*>(o)[i] = r;
        }
    } else {
        for (int i = lane; i < D; i += 32) o[i] = mix_value(alpha, beta, a[i], b[i]);
    }
}

__global__ void __launch_bounds__(ROW_WARPS * 32)
layernorm_kernel(long long n, int D, int vec, const float* __restrict__ in, const float* __restrict__ gamma,
                 float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= n) return;
    const float* src = in + j * D;
    float mean, rstd;
    warp_row_stats(src, D, vec != 0, mean, rstd);
    for (int base = 4 * lane; base < D; base += 128) {
        const float4 v = load_row4(src, base, D, vec != 0);
        const float4 g = load_row4(gamma, base, D, vec != 0);
        const float r[4] = {ln_apply(v.x, mean, rstd, g.x), ln_apply(v.y, mean, rstd, g.y),
                            ln_apply(v.z, mean, rstd, g.z), ln_apply(v.w, mean, rstd, g.w)};
        if (vec) {
            *reinterpret_cast<float4*>(out + j * D + base) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
            for (int k = 0; k < 4 && base + k < D; ++k) out[j * D + base + k] = r[k];
        }
    }
}

// h = LN(x; gamma) for rows already in place, as the scatter kernels write it.
__global__ void __launch_bounds__(ROW_WARPS * 32)
ln_rows_kernel(long long n, int D, int vec, const float* __restrict__ in, const float* __restrict__ gamma,
               float* __restrict__ h) {
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= n) return;
    warp_ln_rows(in + j * D, gamma, D, vec != 0, h + j * (long long)padded_row(D));
}
__global__ void __launch_bounds__(ROW_WARPS * 32)
ln_pack_kernel(long long n, int D, int vec, const float* __restrict__ in, const float* __restrict__ gamma,
               uint16_t* __restrict__ h, float2* __restrict__ row_info) {
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= n) return;
    warp_ln_pack(in + j * D, gamma, D, vec != 0, h + j * (long long)pack_pitch(D), row_info + j);
}

__global__ void gelu_dot_kernel(const float* __restrict__ a, float* __restrict__ b, size_t len) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride) b[i] = gelu_dot(a[i], b[i]);
}

// Weight matrix -> tile-contiguous layout: tiles of 128 rows x 32 values (16 KB),
// tile (mb, kb) at ((mb * KB + kb) * 128 rows; rows and columns past the matrix are zero.  With two sources
// the rows are interleaved: row 2f = src0[f], row 2f+1 = src1[f] (wi_0 / wi_1).  One warp moves one 128-byte
// row segment, so both the read and the write are coalesced.
//
// retile_kernel: raw FP32 tiles for the CUDA-core GEMM.
__global__ void __launch_bounds__(256)
retile_kernel(const float* __restrict__ src0, const float* __restrict__ src1, int M, int K, int MB, int KB,
              float* __restrict__ dst) {
    const int lane = threadIdx.x & 31;
    const long long seg = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);   // (mb, kb, r) flattened
    const long long total = (long long)MB * KB * 128;
    if (seg >= total) return;
    const int r = (int)(seg % 128);
    const long long tile = seg / 128;
    const int kb = (int)(tile % KB), mb = (int)(tile / KB);
    const int m = mb * 128 + r, k = kb * 32 + lane;
    float v = 0.f;
    if (m < M && k < K) {
        if (src1) v = (m & 1) ? src1[(size_t)(m >> 1) * K + k] : src0[(size_t)(m >> 1) * K + k];
        else v = src0[(size_t)m * K + k];
    }
    dst[seg * 32 + lane] = v;
}

// Tensor-core GEMM: both planes of an expert in three launches (an expert that is streamed pays for them on every call).
//
// An FP16 pair holds an FP32 value to its last bit only down to 2^-17 of the largest value under the same power of two
// (split_f16), and there is one power of two per row of an operand.  A layer whose values are uneven inside a row, one
// neuron with large weights or LayerNorm weights of many magnitudes, would lose its small values.  So the layout evens
// the rows out by powers of two that cancel in the products, all exact:
//   per column k of wi_0 / wi_1   2^E_k, E_k the exponent of the column's largest weight, moves from both matrices into
//                                 the LayerNorm weight: gamma'[k] = gamma[k] 2^E_k is what the scatter kernels apply.  h'
//                                 then holds every feature at the size at which it counts in the product, so features
//                                 and columns of any magnitudes that make up for one another are even again
//   per neuron f                  2^a_f moves from column f of wo into g: a_f = max ω - ω_f (+ share), ω_f = log2(|wi_0'[f]|
//                                 |wi_1'[f]|) (2-norms, rounded up).  g_f 2^a_f is at most |h'|^2 2^(max ω) whichever neuron it is
//                                 (g_exponent), and a neuron with large weights no longer sets the scale of all the others.
//                                 2^a_f is part of the 2^-s kept for the rows of wi_1, so the GEMM kernels do nothing for it
//   share                         where neurons remain uneven, ω_f plus the exponent of wo's column f being more than 2^14
//                                 below the largest, half of what is beyond that (at most 2^8) goes back to g: g has a few
//                                 bits to spare, wo 17, and so both keep about the same
// Error against 64 bits of the expert term, worst token, d_model 1024 to 4096 (operands emulated on the CPU; before = one
// scale per row without this; tf32 = TF32 head and BF16 tails): ordinary weights 1.8e-7 (before 1.8e-7, tf32 1.3e-6); one neuron
// x 1000, its wo column / 10^6, 1.8e-7 (1.0e-3, 1.3e-6); LayerNorm weights over 2^-8..2^8, wi inverse, 1.8e-7 (5.9e-2, 1.3e-6); over
// 2^-24..2^24 1.7e-7 (1.0, 1.3e-6); one neuron x 4096, nothing making up for it, 1e-6 to 2e-5 (3e-2 to 1e-1, 3e-5 to 5e-5).
// What remains out of reach: a value more than 2^20 below the largest of its row after all this, in a product to which
// the larger ones contribute nothing (their weights being zero), and a token all of whose gates are more than about 2^18
// below their bound (every weight, feature and row scale log-normal, sigma 2: worst token 3e-4, median 2.5e-7).
constexpr int SHARE_FROM = 14, SHARE_MOST = 8, GAIN_MOST = 64;   // limits of a_f, as exponents
constexpr int W01_EXPONENT_MOST = 110;                           // of a row of wi: 2^-s 2^a_f stays a normal float

struct SplitExpert {
    const float *gamma, *wi0, *wi1, *wo;
    int D, F;
    float *w01, *wo_dst;         // destination planes; behind their tiles:
    float *inv01, *inv_wo;       // 2^-s of every padded row (wi_1 rows: times 2^a_f)
    int* range;                  // max over f of ω_f and of ω_f + exponent of wo's column f
    int* omega;                  // ω_f
    int *col01, *col_wo;         // exponent of the largest weight of every padded column
    float* gamma_out;            // gamma'
    int KB01, KBwo;              // 32-column blocks
};

// biased exponent; of a zero: below that of any other value under any shift
__device__ __forceinline__ int exponent_field(float x) {
    const int u = __float_as_int(x) & 0x7fffffff;
    return u ? u >> 23 : -4000;
}
// x 2^e for any e that two normal factors make up; exact unless the result is below the normal range
__device__ __forceinline__ float scale_by(float x, int e) {
    const int half = e >> 1;
    return __fmul_rn(__fmul_rn(x, exp2_int(half)), exp2_int(e - half));
}
__device__ __forceinline__ float4 load4(const float* __restrict__ p, bool vec) {
    return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}

// Column exponents.  A cluster of eight blocks per 32 columns, eight lanes to a row (four columns each), the rows dealt out
// over the cluster's 256 such groups; the blocks' maxima meet in the first one through distributed shared memory, so
// nothing has to be zeroed first.  Bound by HBM (each weight is read once).  Magnitudes are compared as integers, so
// NaN counts as the largest.
constexpr int COL_CLUSTER = 8;
__global__ void __launch_bounds__(256) __cluster_dims__(COL_CLUSTER, 1, 1)
column_exponent_kernel(const SplitExpert a, int vec) {
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ uint32_t s_warp[8][32];
    __shared__ uint32_t s_block[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = (int)cluster.block_rank();
    int slab = (int)blockIdx.x / COL_CLUSTER;
    const bool wo = slab >= a.KB01;
    if (wo) slab -= a.KB01;
    const int K = wo ? a.F : a.D, rows = wo ? a.D : a.F, k = slab * 32 + 4 * (lane & 7);
    const int first = (rank * 256 + (int)threadIdx.x) >> 3;
    uint32_t top[4] = {0, 0, 0, 0};
    const auto take = [&](const float4 v) {
        top[0] = max(top[0], __float_as_uint(v.x) & 0x7fffffffu);
        top[1] = max(top[1], __float_as_uint(v.y) & 0x7fffffffu);
        top[2] = max(top[2], __float_as_uint(v.z) & 0x7fffffffu);
        top[3] = max(top[3], __float_as_uint(v.w) & 0x7fffffffu);
    };
    pdl_trigger();
    if (k < K) {                                               // K is a multiple of 4
        if (wo) {
#pragma unroll 8
            for (int r = first; r < rows; r += 32 * COL_CLUSTER) take(load4(a.wo + (size_t)r * K + k, vec != 0));
        } else {
#pragma unroll 4
            for (int r = first; r < rows; r += 32 * COL_CLUSTER) {
                const float4 v0 = load4(a.wi0 + (size_t)r * K + k, vec != 0), v1 = load4(a.wi1 + (size_t)r * K + k, vec != 0);
                take(v0);
                take(v1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        top[i] = max(top[i], __shfl_xor_sync(0xffffffffu, top[i], 8));
        top[i] = max(top[i], __shfl_xor_sync(0xffffffffu, top[i], 16));
        if (lane < 8) s_warp[warp][4 * lane + i] = top[i];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t best = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) best = max(best, s_warp[w][lane]);
        s_block[lane] = best;
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x < 32) {
        const int column = slab * 32 + lane;
        uint32_t best = 0;
#pragma unroll
        for (int q = 0; q < COL_CLUSTER; ++q) best = max(best, cluster.map_shared_rank(s_block, q)[lane]);
        const int field = (int)(best >> 23);
        const int e = column < K && field < 255 ? max(field - 127, -126) : 0;     // infinities and NaN move nothing
        (wo ? a.col_wo : a.col01)[column] = e;
        if (!wo) a.gamma_out[column] = column < K ? __fmul_rn(a.gamma[column], exp2_int(e)) : 0.f;
    }
    if (blockIdx.x == 0 && threadIdx.x < 2) a.range[threadIdx.x] = INT_MIN;
    cluster.sync();                                            // no block leaves while its maxima can still be read
}

// a_f from ω_f, the exponent of wo's column f and the two maxima.
__device__ __forceinline__ int neuron_gain(int omega, int column, int max_omega, int max_reach) {
    const int below = max_reach - (omega + column);
    const int share = below > SHARE_FROM ? min((below - SHARE_FROM + 1) / 2, SHARE_MOST) : 0;
    return min(max(max_omega - omega - share, -SHARE_MOST), GAIN_MOST);
}

// ROWS weight rows side by side, their elements times 2^-shift[k], to FP16 pairs in their rows of the tiles (a row of a tile
// being 32 x hi, 32 x lo), each scaled by 2^s so that its largest magnitude lands in [2^14, 2^15).  `squares` are the sums
// of squares of the scaled rows.  WARPS warps of the block share the rows, 128 columns at a time: a lane holds four
// neighbouring values, so a warp reads 512 bytes and writes four whole 128-byte rows.  The rows are read twice, the second
// time from L1 or L2.  in = false: rows of zeros.  Bound by HBM for large experts, by latency for small ones.  Rows are few and
// long or many and short, and WARPS makes up about as many warps either way.  Columns, w01, wo, us: 4096 x 10240 85, 168, 112;
// 1024 x 4096 14, 17, 15; 160 x 600 5.7, 4.6, 5.3.  A whole set_expert at 1024 x 4096: 103 with one warp per row and eight
// blocks per 128 columns, now 63 (60 without the column scales).
template <int ROWS, int WARPS, typename Shift>
__device__ __forceinline__ void split_rows(const float* const (&row)[ROWS], bool in, int K, int KB, bool vec, int most,
                                           uint32_t* const (&dst)[ROWS], const Shift& shift, int (&s)[ROWS],
                                           float (&squares)[ROWS]) {
    __shared__ int s_top[8][ROWS];
    __shared__ float s_squares[8][ROWS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % WARPS, group = warp / WARPS * WARPS;
    constexpr int INFINITE = 4000;
    int top[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) top[i] = -4000;
    if (in) {
#pragma unroll 4
        for (int k = 4 * lane + 128 * part; k < K; k += 128 * WARPS) {
            float4 v[ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i) v[i] = load4(row[i] + k, vec);
            const int4 c = shift(k);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int f0 = exponent_field(v[i].x), f1 = exponent_field(v[i].y), f2 = exponent_field(v[i].z),
                          f3 = exponent_field(v[i].w);
                top[i] = max(max(max(top[i], f0 - c.x), max(f1 - c.y, f2 - c.z)), f3 - c.w);
                if (max(max(f0, f1), max(f2, f3)) == 255) top[i] = INFINITE;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        top[i] = __reduce_max_sync(0xffffffffu, top[i]);
        if (WARPS > 1 && lane == 0) s_top[warp][i] = top[i];
    }
    if (WARPS > 1) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
            for (int w = 0; w < WARPS; ++w) top[i] = max(top[i], s_top[group + w][i]);
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        // a row with an infinity or a NaN only has to hand it on; a row of zeros takes any scale
        s[i] = !in || top[i] == INFINITE ? 0 : min(max(14 + 127 - top[i], -126), most);
        squares[i] = 0.f;
    }
#pragma unroll 2
    for (int k = 4 * lane + 128 * part; k < KB * 32; k += 128 * WARPS) {
        float4 w[ROWS];
        int4 c = make_int4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) w[i] = in && k < K ? load4(row[i] + k, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (in && k < K) c = shift(k);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float v[4] = {scale_by(w[i].x, s[i] - c.x), scale_by(w[i].y, s[i] - c.y), scale_by(w[i].z, s[i] - c.z),
                                scale_by(w[i].w, s[i] - c.w)};
#pragma unroll
            for (int j = 0; j < 4; ++j) squares[i] = fmaf(v[j], v[j], squares[i]);
            store_pack4(reinterpret_cast<uint16_t*>(dst[i] + (size_t)(k >> 5) * 4096), k & 31, v);
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        squares[i] = warp_xor_sum(squares[i]);
        if (WARPS > 1 && lane == 0) s_squares[warp][i] = squares[i];
    }
    if (WARPS > 1) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            squares[i] = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) squares[i] += s_squares[group + w][i];
        }
    }
}

// w01: WARPS warps per neuron f, the rows 2 f = wi_0[f] and 2 f + 1 = wi_1[f].
template <int WARPS>
__global__ void __launch_bounds__(256)
split_w01_kernel(const SplitExpert a, int vec) {
    __shared__ int s_omega[8], s_reach[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = ((int)blockIdx.x * 8 + warp) / WARPS;        // the grid covers the padded rows exactly
    pdl_trigger();
    pdl_wait();
    const auto shift = [&](int k) { return *reinterpret_cast<const int4*>(a.col01 + k); };
    const bool in = f < a.F;
    const float* const row[2] = {a.wi0 + (size_t)f * a.D, a.wi1 + (size_t)f * a.D};
    uint32_t* const dst0 = reinterpret_cast<uint32_t*>(a.w01) + (size_t)(f >> 6) * a.KB01 * 4096 + (size_t)(f & 63) * 64;
    uint32_t* const dst[2] = {dst0, dst0 + 32};
    float squares[2];
    int s[2];
    split_rows<2, WARPS>(row, in, a.D, a.KB01, vec != 0, W01_EXPONENT_MOST, dst, shift, s, squares);
    if (lane == 0) {
        int omega = -1000, reach = -1000;
        if (in) {
            const float w = 0.5f * (log2f(squares[0]) + log2f(squares[1])) - (float)(s[0] + s[1]) + 0.01f;
            omega = w > -400.f ? (int)ceilf(fminf(w, 400.f)) : -400;    // a row of zeros, or a NaN
            reach = omega + a.col_wo[f];
            a.omega[f] = omega;
        }
        a.inv01[2 * f] = exp2_int(-s[0]);
        a.inv01[2 * f + 1] = exp2_int(-s[1]);                  // times 2^a_f in the next launch
        s_omega[warp] = omega;
        s_reach[warp] = reach;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) {
            s_omega[0] = max(s_omega[0], s_omega[i]);
            s_reach[0] = max(s_reach[0], s_reach[i]);
        }
        atomicMax(a.range, s_omega[0]);
        atomicMax(a.range + 1, s_reach[0]);
    }
}

// wo: WARPS warps per row; the blocks behind those of the rows multiply 2^a_f into 2^-s of wi_1's rows.
template <int WARPS>
__global__ void __launch_bounds__(256)
split_wo_kernel(const SplitExpert a, int vec, int row_blocks) {
    pdl_trigger();
    pdl_wait();
    const int max_omega = a.range[0], max_reach = a.range[1];
    if ((int)blockIdx.x >= row_blocks) {
        const int f = ((int)blockIdx.x - row_blocks) * 256 + (int)threadIdx.x;
        if (f < a.F)
            a.inv01[2 * f + 1] = __fmul_rn(a.inv01[2 * f + 1], exp2_int(neuron_gain(a.omega[f], a.col_wo[f], max_omega, max_reach)));
        return;
    }
    const int r = ((int)blockIdx.x * 8 + (int)(threadIdx.x >> 5)) / WARPS;
    const auto shift = [&](int k) {
        const int4 w = *reinterpret_cast<const int4*>(a.omega + k), c = *reinterpret_cast<const int4*>(a.col_wo + k);
        return make_int4(neuron_gain(w.x, c.x, max_omega, max_reach), neuron_gain(w.y, c.y, max_omega, max_reach),
                         neuron_gain(w.z, c.z, max_omega, max_reach), neuron_gain(w.w, c.w, max_omega, max_reach));
    };
    const float* const row[1] = {a.wo + (size_t)r * a.F};
    uint32_t* const dst[1] = {reinterpret_cast<uint32_t*>(a.wo_dst) + (size_t)(r >> 7) * a.KBwo * 4096 + (size_t)(r & 127) * 32};
    float unused[1];
    int s[1];
    split_rows<1, WARPS>(row, r < a.D, a.F, a.KBwo, vec != 0, 126, dst, shift, s, unused);
    if ((threadIdx.x & 31) == 0) a.inv_wo[r] = exp2_int(-s[0]);
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
inline unsigned row_grid(long long rows) { return (unsigned)((rows + ROW_WARPS - 1) / ROW_WARPS); }

}  // namespace

int launch_scatter(long long T, int D, const float* X, const float* coeff, const int* pos, float* routed,
                   float* rcoeff, cudaStream_t stream) {
    if (T < 0 || D <= 0 || !X || !pos || !routed) {
        set_error("expert_scatter: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (T == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(X) && aligned16(routed);
    INFMOE_CUDA_TRY(launch_chained(scatter_kernel, row_grid(T), ROW_WARPS * 32, 0, 1, stream, T, D, vec, X, coeff, pos,
                                   routed, rcoeff));
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

// Up to 1024 tokens whose row and LayerNorm weight fit into 48 KB of shared memory with the histogram's E + 1 words; up to
// DM_MAX_TOKENS of aligned rows that eight warps hold in registers.
bool dispatch_scatter_supported(long long T, int D, int E, const float* X, bool pack) {
    if (E >= 8192) return false;
    if (T <= 1024 && D <= 6016) return true;
    return pack && T <= DM_MAX_TOKENS && D <= 2048 && D % 4 == 0 && aligned16(X);
}

int launch_dispatch_scatter(long long T, int D, int E, const float* X, const float* score, const int* gate,
                            const float* gamma, size_t gamma_stride, int* pos, int* count, int* offset, int* status,
                            int* zero, int zero_count, float* rscore, void* h, float* row_info, bool pack, bool early,
                            cudaStream_t stream) {
    const int vec = (D % 4 == 0) && (gamma_stride % 4 == 0) && aligned16(X) && aligned16(gamma);
    const ExpertGamma gammas{gamma, gamma_stride};
    const size_t hist = sizeof(int) * (size_t)(E + 1);
    if (!zero) zero_count = 0;
    if (T <= 1024 && D <= 6016) {
        size_t smem = 2 * padded_row(D) * sizeof(float);
        if (smem < hist) smem = hist;
        auto kern = pack ? dispatch_scatter_kernel<true> : dispatch_scatter_kernel<false>;
        INFMOE_CUDA_TRY(launch_chained(kern, (unsigned)T + 1, DS_THREADS, smem, 1, stream, (int)T, D, E, vec, X, score, gate,
                                       gammas, pos, count, offset, status, zero, zero_count, rscore, h, (float2*)row_info,
                                       early ? 1 : 0));
    } else {
        if (!vec || !pack) {
            set_error("dispatch_scatter: unaligned rows");
            return INFMOE_ERR_UNSUPPORTED;
        }
        const int nv = D <= 512 ? 4 : D <= 1024 ? 8 : 16;
        size_t smem = (size_t)DM_TOKENS * nv * 512;
        if (smem < hist) smem = hist;
        auto kern = nv == 4 ? dispatch_scatter_reg_kernel<4>
                            : nv == 8 ? dispatch_scatter_reg_kernel<8> : dispatch_scatter_reg_kernel<16>;
        if (smem > 48 * 1024)
            INFMOE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        INFMOE_CUDA_TRY(launch_chained(kern, (unsigned)((T + DM_TOKENS - 1) / DM_TOKENS + 1), DM_THREADS, smem, 1, stream,
                                       (int)T, D, E, X, score, gate, gammas, pos, count, offset, status, zero, zero_count,
                                       rscore, (uint16_t*)h, (float2*)row_info, early ? 1 : 0));
    }
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_scatter_ln_rows(long long T, int D, const float* X, const float* score, const int* pos, const int* gate,
                           const float* gamma_all, const int* valid_rows, float* rscore, float* h, cudaStream_t stream) {
    if (T == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(X) && aligned16(gamma_all);
    INFMOE_CUDA_TRY(launch_chained(scatter_ln_rows_kernel, row_grid(T), ROW_WARPS * 32, 0, 1, stream, T, D, vec, X, score,
                                   pos, gate, gamma_all, valid_rows, rscore, h));
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_scatter_ln_pack(long long row0, long long T, int D, const float* X, const float* score, const int* pos,
                           const int* gate, const float* gamma, size_t gamma_stride, const int* valid_rows, float* rscore,
                           void* h, float* row_info, cudaStream_t stream) {
    if (T == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && (gamma_stride % 4 == 0) && aligned16(X) && aligned16(gamma);
    const ExpertGamma gammas{gamma, gamma_stride};
    uint16_t* pack = (uint16_t*)h;
    float2* info = (float2*)row_info;
    if (vec && D <= 4096) {
        const unsigned grid = (unsigned)((T + 3) / 4);
#define INFMOE_SCATTER_REG(NV)                                                                                     \
    do {                                                                                                           \
        auto kern = scatter_ln_pack_reg_kernel<NV>;                                                                \
        constexpr int smem = 4 * NV * 32 * 16;                                                                     \
        if (smem > 48 * 1024)                                                                                      \
            INFMOE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));        \
        INFMOE_CUDA_TRY(launch_chained(kern, grid, 128, smem, 1, stream, row0, T, D, X, score, pos, gate, gammas,  \
                                       valid_rows, rscore, pack, info));                                           \
    } while (0)
        if (D <= 1024) INFMOE_SCATTER_REG(8);
        else if (D <= 2048) INFMOE_SCATTER_REG(16);
        else INFMOE_SCATTER_REG(32);
#undef INFMOE_SCATTER_REG
    } else {
        INFMOE_CUDA_TRY(launch_chained(scatter_ln_pack_kernel, row_grid(T), ROW_WARPS * 32, 0, 1, stream, row0, T, D, vec, X,
                                       score, pos, gate, gammas, valid_rows, rscore, pack, info));
    }
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

namespace {
// in[i,:] -> the row at address dst[i]
__global__ void __launch_bounds__(ROW_WARPS * 32)
rows_to_ptrs_kernel(long long n, int D, int vec, const float* __restrict__ in, const unsigned long long* __restrict__ dst) {
    const int lane = threadIdx.x & 31;
    const long long j = (long long)blockIdx.x * ROW_WARPS + (threadIdx.x >> 5);
    if (j >= n) return;
    const float* a = in + j * D;
    float* o = reinterpret_cast<float*>(dst[j]);
    if (vec && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
        for (int i = lane; i < D / 4; i += 32) reinterpret_cast<float4*>(o)[i] = reinterpret_cast<const float4*>(a)[i];
    } else {
        for (int i = lane; i < D; i += 32) o[i] = a[i];
    }
}
}  // namespace

int launch_rows_to_ptrs(long long n, int D, const float* in, const unsigned long long* dst, cudaStream_t stream) {
    if (n < 0 || D <= 0 || !in || !dst) {
        set_error("rows_to_ptrs: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (n == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(in);
    rows_to_ptrs_kernel<<<row_grid(n), ROW_WARPS * 32, 0, stream>>>(n, D, vec, in, dst);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_gather(long long T, int D, const float* in, const int* pos, float* out, cudaStream_t stream,
                  const int* valid_rows) {
    if (T < 0 || D <= 0 || !in || !pos || !out) {
        set_error("expert_gather: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (T == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(in) && aligned16(out);
    INFMOE_CUDA_TRY(launch_chained(gather_kernel, row_grid(T), ROW_WARPS * 32, 0, 1, stream, T, D, vec, in, pos, valid_rows,
                                   out));
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_mix_gather(long long T, int D, const int* pos, const float* routed, const float* post,
                      const float* coeff, float* out, cudaStream_t stream, const int* valid_rows) {
    if (T < 0 || D <= 0 || !pos || !routed || !post || !coeff || !out) {
        set_error("expert_mix_gather: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (T == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(routed) && aligned16(post) && aligned16(out);
    INFMOE_CUDA_TRY(launch_chained(mix_gather_kernel, row_grid(T), ROW_WARPS * 32, 0, 1, stream, T, D, vec, pos, routed, post,
                                   coeff, valid_rows, out));
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_layernorm(float* out, const float* in, long long n, int D, const float* gamma, cudaStream_t stream) {
    if (n < 0 || D <= 0 || !out || !in || !gamma) {
        set_error("layernorm: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (n == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(in) && aligned16(out) && aligned16(gamma);
    layernorm_kernel<<<row_grid(n), ROW_WARPS * 32, 0, stream>>>(n, D, vec, in, gamma, out);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_ln_rows(long long n, int D, const float* in, const float* gamma, float* h, cudaStream_t stream) {
    if (n == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(in) && aligned16(gamma);
    ln_rows_kernel<<<row_grid(n), ROW_WARPS * 32, 0, stream>>>(n, D, vec, in, gamma, h);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_ln_pack(long long n, int D, const float* in, const float* gamma, void* h, float* row_info,
                   cudaStream_t stream) {
    if (n == 0) return INFMOE_OK;
    const int vec = (D % 4 == 0) && aligned16(in) && aligned16(gamma);
    ln_pack_kernel<<<row_grid(n), ROW_WARPS * 32, 0, stream>>>(n, D, vec, in, gamma, (uint16_t*)h, (float2*)row_info);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_split_expert(const float* gamma, const float* wi0, const float* wi1, const float* wo, int D, int F, float* w01,
                        float* wo_dst, cudaStream_t stream) {
    SplitExpert a;
    a.gamma = gamma;
    a.wi0 = wi0;
    a.wi1 = wi1;
    a.wo = wo;
    a.D = D;
    a.F = F;
    a.w01 = w01;
    a.wo_dst = wo_dst;
    a.inv01 = w01 + tiled_elems(2 * F, D);
    a.inv_wo = wo_dst + tiled_elems(D, F);
    a.range = (int*)(w01 + split_range_at(2 * F, D));
    a.omega = a.range + 32;
    a.col01 = (int*)(w01 + split_columns_at(2 * F, D));
    a.col_wo = (int*)(wo_dst + split_columns_at(D, F));
    a.gamma_out = w01 + split_gamma_at(2 * F, D);
    a.KB01 = (D + 31) / 32;
    a.KBwo = (F + 31) / 32;
    const int vec = aligned16(wi0) && aligned16(wi1) && aligned16(wo);     // D and F are multiples of 4
    column_exponent_kernel<<<(unsigned)((a.KB01 + a.KBwo) * COL_CLUSTER), 256, 0, stream>>>(a, vec);
    INFMOE_CUDA_TRY(cudaGetLastError());
    // one to eight warps per row: up to about 8000 of them, at least one step of 128 columns each
    const auto warps_per_row = [](int rows, int K) {
        int w = 1;
        while (w < 8 && rows * w * 2 <= 8192 && w * 2 * 128 <= K + 127) w *= 2;
        return w;
    };
    const int neurons = (2 * F + 127) / 128 * 64, rows = (D + 127) / 128 * 128;
    const int w1 = warps_per_row(neurons, D), w2 = warps_per_row(rows, F), row_blocks = rows * w2 / 8;
    auto k1 = w1 == 1 ? split_w01_kernel<1> : w1 == 2 ? split_w01_kernel<2> : w1 == 4 ? split_w01_kernel<4> : split_w01_kernel<8>;
    auto k2 = w2 == 1 ? split_wo_kernel<1> : w2 == 2 ? split_wo_kernel<2> : w2 == 4 ? split_wo_kernel<4> : split_wo_kernel<8>;
    INFMOE_CUDA_TRY(launch_chained(k1, (unsigned)(neurons * w1 / 8), 256, 0, 1, stream, a, vec));
    INFMOE_CUDA_TRY(launch_chained(k2, (unsigned)(row_blocks + (F + 255) / 256), 256, 0, 1, stream, a, vec, row_blocks));
    note_launch(3);
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_retile(const float* src0, const float* src1, int M, int K, float* dst, cudaStream_t stream) {
    const int MB = (M + 127) / 128, KB = (K + 31) / 32;
    const long long segs = (long long)MB * KB * 128;
    retile_kernel<<<(unsigned)((segs + 7) / 8), 256, 0, stream>>>(src0, src1, M, K, MB, KB, dst);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

int launch_gelu_dot(const float* a, float* b, size_t len, cudaStream_t stream) {
    if (!a || !b) {
        set_error("gelu_dot: bad argument");
        return INFMOE_ERR_INVALID_ARGUMENT;
    }
    if (len == 0) return INFMOE_OK;
    const unsigned grid = (unsigned)((len + 255) / 256 < 148 * 16 ? (len + 255) / 256 : 148 * 16);
    gelu_dot_kernel<<<grid, 256, 0, stream>>>(a, b, len);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

namespace {
__global__ void fill_int_kernel(int* dst, int value) { *dst = value; }
}  // namespace

int launch_fill_int(int* dst, int value, cudaStream_t stream) {
    fill_int_kernel<<<1, 1, 0, stream>>>(dst, value);
    note_launch();
    INFMOE_CUDA_TRY(cudaGetLastError());
    return INFMOE_OK;
}

}  // namespace infmoe
