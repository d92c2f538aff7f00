// Shared host/device helpers of the B200 MoE-layer kernels.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>
#include <cstdio>

#include "infmoe_c.h"

namespace infmoe {

// ---------------------------------------------------------------------------
// Error plumbing: nothing in this library exits the process (the reference's
// CUDA_SAFE_CALL does, plugin/utility.h:15-21); every failure becomes a status.
// ---------------------------------------------------------------------------
void set_error(const char* fmt, ...) __attribute__((format(printf, 1, 2)));

#define INFMOE_CUDA_TRY(call)                                                                              \
    do {                                                                                                   \
        cudaError_t err__ = (call);                                                                        \
        if (err__ != cudaSuccess) {                                                                        \
            ::infmoe::set_error("CUDA error %d (%s) at %s:%d", (int)err__, cudaGetErrorString(err__),      \
                                __FILE__, __LINE__);                                                       \
            return INFMOE_ERR_CUDA;                                                                        \
        }                                                                                                  \
    } while (0)

#define INFMOE_TRY(call)                \
    do {                                \
        int rc__ = (call);              \
        if (rc__ != INFMOE_OK) return rc__; \
    } while (0)

// Bits of the device-side status word.
enum : int32_t {
    STATUS_NO_EXPERT = 1,      // a token selected no expert (NaN scores)
    STATUS_BAD_GATE = 2,       // gate index outside [0, E)
    STATUS_WAIT_TIMEOUT = 4,   // a bounded mbarrier wait ran out inside a GEMM kernel
    STATUS_BAD_SHAPE = 8,
};

// Process-wide count of kernels launched by this library.
extern long long g_kernel_launches;
inline void note_launch(int n = 1) { g_kernel_launches += n; }

#ifdef __CUDACC__
// Launches a kernel that begins with pdl_wait (see there); cluster > 1: in clusters of that many blocks.
template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kern)(Params...), unsigned grid, unsigned threads, size_t smem, unsigned cluster,
                                  cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, Params(args)...);
}

// ---------------------------------------------------------------------------
// Programmatic dependent launch.  The kernels of a pass are short next to the time between two dependent launches
// (1-2 us on an idle GPU), so each is launched while its predecessor still runs (launch_chained): its blocks start as
// soon as every block of the predecessor has called pdl_trigger and left room, do what needs no memory, and wait
// in pdl_wait until the predecessor has completed and its writes are visible.  Every block of every kernel launched
// this way calls pdl_wait, and writes no global memory before it; the predecessor did the same, so all earlier kernels of the
// stream are complete then too.  (Without the launch attribute both are no-ops.)
// What may be read before the wait: what no kernel on the stream writes (the routing reads centroids and LayerNorm weights so),
// and, behind a predecessor that calls pdl_trigger only after its own wait, what was complete when that one's wait ended.
// Routing, dispatch and scatter kernels all trigger so: the scatters read the tokens, the first GEMM gates or offsets and
// weights; it does too, for the second one.  The others (second GEMM, combine, weight layout) trigger first, and a kernel behind
// them reads nothing of the second kind.
// Nothing that a predecessor may still be writing is read
// through the read-only path: `const T* __restrict__` parameters and __ldg promise that nobody writes during the kernel, and a
// load under that promise may be moved above the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Canonical FP32 reductions.  Routing must agree bit for bit with the CPU
// checker, so the summation order is fixed: lane l of a warp owns elements
// k = 4*(l + 32*i) + c (i ascending, c = 0..3), accumulates them in that order
// with explicit round-to-nearest adds / fused multiply-adds, and the 32 lane
// partials are combined by a butterfly (xor 16, 8, 4, 2, 1).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float warp_xor_sum(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// Loads elements [base, base+4) of a row; `vec` says the row is 16-byte aligned
// with D % 4 == 0.  Elements at or beyond D read as 0 and must be skipped by the caller.
__device__ __forceinline__ float4 load_row4(const float* __restrict__ row, int base, int D, bool vec) {
    if (vec) return *reinterpret_cast<const float4*>(row + base);
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (base + 0 < D) r.x = row[base + 0];
    if (base + 1 < D) r.y = row[base + 1];
    if (base + 2 < D) r.z = row[base + 2];
    if (base + 3 < D) r.w = row[base + 3];
    return r;
}

// LayerNorm statistics of one row held by a full warp (true LayerNorm: mean
// subtracted, biased variance, eps 1e-6; reference plugin/cuda/ops/layernorm.cu:126-149).
__device__ __forceinline__ void warp_row_stats(const float* __restrict__ row, int D, bool vec, float& mean,
                                               float& rstd) {
    const int lane = threadIdx.x & 31;
    // Same additions in the same order either way; the vector form (D a multiple of 4, aligned rows) has no
    // per-element bounds checks and keeps eight loads in flight.
    float s = 0.f;
    if (vec) {
#pragma unroll 8
        for (int base = 4 * lane; base < D; base += 128) {
            const float4 v = *reinterpret_cast<const float4*>(row + base);
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
        }
    } else {
        for (int base = 4 * lane; base < D; base += 128) {
            const float4 v = load_row4(row, base, D, false);
            s = __fadd_rn(s, v.x);
            if (base + 1 < D) s = __fadd_rn(s, v.y);
            if (base + 2 < D) s = __fadd_rn(s, v.z);
            if (base + 3 < D) s = __fadd_rn(s, v.w);
        }
    }
    mean = __fdiv_rn(warp_xor_sum(s), (float)D);
    float q = 0.f;
    if (vec) {
#pragma unroll 8
        for (int base = 4 * lane; base < D; base += 128) {
            const float4 v = *reinterpret_cast<const float4*>(row + base);
            float d = __fsub_rn(v.x, mean);
            q = __fmaf_rn(d, d, q);
            d = __fsub_rn(v.y, mean);
            q = __fmaf_rn(d, d, q);
            d = __fsub_rn(v.z, mean);
            q = __fmaf_rn(d, d, q);
            d = __fsub_rn(v.w, mean);
            q = __fmaf_rn(d, d, q);
        }
    } else {
        for (int base = 4 * lane; base < D; base += 128) {
            const float4 v = load_row4(row, base, D, false);
            float d = __fsub_rn(v.x, mean);
            q = __fmaf_rn(d, d, q);
            if (base + 1 < D) { d = __fsub_rn(v.y, mean); q = __fmaf_rn(d, d, q); }
            if (base + 2 < D) { d = __fsub_rn(v.z, mean); q = __fmaf_rn(d, d, q); }
            if (base + 3 < D) { d = __fsub_rn(v.w, mean); q = __fmaf_rn(d, d, q); }
        }
    }
    const float var = __fdiv_rn(warp_xor_sum(q), (float)D);
    rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var, 1e-6f)));
}

// gamma * ((x - mean) * rstd), reference plugin/cuda/ops/layernorm.cu:158-161.
__device__ __forceinline__ float ln_apply(float x, float mean, float rstd, float gamma) {
    return __fmul_rn(gamma, __fmul_rn(__fsub_rn(x, mean), rstd));
}

// Operand of the tensor-core GEMM: an FP32 value, scaled by powers of two of its row and column, as a pair of FP16 values,
// hi = x rounded to 11 significant bits, lo = x - hi rounded to 11 (in the lower / upper half of the word).  |lo| is at
// most half a unit of hi, so together they hold x to within 2^-23 relative (the last bit of an FP32 value) down to
// |x| = 2^-2, which is 2^-17 of the row's largest value.  Below that FP16's smallest step sets an absolute limit, 2^-25, so
// rows have to be even; see the weight layout in rows.cu.
__device__ __forceinline__ uint32_t split_f16(float x) {
    const __half hi = __float2half_rn(x);
    const __half lo = __float2half_rn(__fsub_rn(x, __half2float(hi)));
    return (uint32_t)__half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16);
}
// Rows of pairs are stored in 128-byte groups of 32 values: 32 x hi followed by 32 x lo; rows are padded with zeros to
// a multiple of 32 values.
__host__ __device__ __forceinline__ size_t pack_pitch(int K) { return (size_t)((K + 31) / 32) * 64; }   // in 16-bit elements
// Floats of a padded FP32 row (CUDA-core GEMM).
__host__ __device__ __forceinline__ size_t padded_row(int K) { return (size_t)((K + 31) / 32) * 32; }
// Stores four consecutive values k0..k0+3 (k0 a multiple of 4) of one row.
__device__ __forceinline__ void store_pack4(uint16_t* __restrict__ pack_row, int k0, const float v[4]) {
    uint16_t* g = pack_row + (size_t)(k0 >> 5) * 64 + (k0 & 31);
    const uint32_t a = split_f16(v[0]), b = split_f16(v[1]), c = split_f16(v[2]), d = split_f16(v[3]);
    *reinterpret_cast<uint2*>(g) = make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(c, d, 0x5410));
    *reinterpret_cast<uint2*>(g + 32) = make_uint2(__byte_perm(a, b, 0x7632), __byte_perm(c, d, 0x7632));
}
// 2^e as a float, e in [-126, 127].
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }
// Exponent s that brings the largest magnitude of a row into [2^14, 2^15) (FP16 ends at 65504); 0 for a row of zeros
// or with an infinity.  At most 126, so that 2^s and 2^-s are both normal floats.
__device__ __forceinline__ int row_exponent(float max_abs) {
    if (!(max_abs > 0.f) || !(max_abs <= FLT_MAX)) return 0;
    return min(126, 14 - ((__float_as_int(max_abs) >> 23) - 127));
}
// Exponent of the gate activations g of one token.  |g_f| = |gelu(a_f) b_f| <= |a_f| |b_f| <= |h|^2 |wi_0[f]| |wi_1[f]|
// (2-norms), and the weight layout scales neuron f by 2^a_f so that |wi_0[f]| |wi_1[f]| 2^a_f <= 2^w for all of them.  So
// with h2 = log2 |h|^2 no g 2^a_f 2^s exceeds 2^15.  The bound is about 2^13 above a typical g at d_model 4096, which
// leaves typical values near 2^2, with all their bits.  Both GEMMs compute it from the same two numbers.
__device__ __forceinline__ int g_exponent(float h2, float w) {
    float b = h2 + w + 0.01f;
    if (!(b > -111.f)) b = -111.f;
    if (!(b < 141.f)) b = 141.f;
    return 15 - (int)ceilf(b);
}
// sum 2^-s of the weight row 2^-s of the token row; the smaller factor first, so that nothing overflows on the way.
__device__ __forceinline__ float unscale(float sum, float w_inv, float x_inv) {
    return __fmul_rn(__fmul_rn(sum, fminf(w_inv, x_inv)), fmaxf(w_inv, x_inv));
}
// Row statistics the tensor-core path keeps of a token row: 2^-s and log2 of the squared norm, from the exponent and
// the sum of squares of the row times 2^s.
__device__ __forceinline__ float2 token_row_info(int s, float scaled_square_sum) {
    return make_float2(exp2_int(-s), scaled_square_sum > 0.f ? log2f(scaled_square_sum) - 2.f * (float)s : -300.f);
}

// base_layer output mix (plugin/cuda/moe.cu:115-127, sigmoid plugin/cuda/common.cuh:24-27):
// out = alpha * expert_output + (1 - alpha) * input with alpha = sigmoid(score).  One fixed rounding sequence, so
// that the stand-alone combine kernel and the GEMM epilogue that fuses it give the same bits.
__device__ __forceinline__ float mix_alpha(float score) { return 1.0f / (1.0f + expf(-score)); }
__device__ __forceinline__ float mix_value(float alpha, float beta, float post, float routed) {
    return __fmaf_rn(alpha, post, __fmul_rn(beta, routed));
}

// gelu(a) * b in the reference's evaluation order (plugin/cuda/ops/gelu.cu:8-15).
__device__ __forceinline__ float gelu_dot(float a, float b) {
    const float cdf = 0.5f * (1.0f + tanhf(a * (0.035677408136300125f * a * a + 0.7978845608028654f)));
    return a * cdf * b;
}
// The same function with 0.5 (1 + tanh(u)) written as the logistic 1 / (1 + exp(-2u)): a handful of instructions
// instead of tanhf's few dozen, for the tensor-core path, whose results are held to a tolerance rather than to the
// reference's bits.  ex2.approx and the approximate division are each good to 2 ulp; for u so negative that
// exp(-2u) overflows the quotient is 0, which is the limit.
__device__ __forceinline__ float gelu_dot_fast(float a, float b) {
    const float u = a * (0.035677408136300125f * a * a + 0.7978845608028654f);
    const float cdf = __fdividef(1.0f, 1.0f + __expf(-2.0f * u));
    return a * cdf * b;
}
#endif  // __CUDACC__

}  // namespace infmoe
