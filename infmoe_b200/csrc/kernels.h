// Launchers of the CUDA kernels (defined in route.cu, dispatch.cu, rows.cu, ffn_simt.cu, ffn_umma.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>

namespace infmoe {

// constant: no kernel or copy that may still be running writes C or gamma, so they may be read before the stream's earlier
// kernels have ended.
int launch_route(const float* X, const float* C, const float* gamma, long long T, int D, int E, int* gate,
                 float* score, int* status, cudaStream_t stream, bool constant = false);
int make_f32_row_map(CUtensorMap* map, const void* base, long long K, long long rows, int box_rows);
int launch_select_top1(long long T, int E, const float* aff, int* gate, float* weight, int* status,
                       cudaStream_t stream);
// region_count != NULL: the T slots are regions of region_size slots, of which only the first region_count[s]
// hold rows (receive buffer of the expert-parallel path); the other slots are skipped silently.
// zero[0 .. zero_count) (may be NULL) is cleared on the way: the counters of the GEMMs' cut tiles.
int launch_dispatch(const int* gate, long long T, int E, int* pos, int* count, int* offset, int* status,
                    cudaStream_t stream, const int* region_count = nullptr, int region_size = 0, int* zero = nullptr,
                    int zero_count = 0);
bool dispatch_supported(int E);   // the expert count fits the dispatch kernel
int launch_scatter(long long T, int D, const float* X, const float* coeff, const int* pos, float* routed,
                   float* rcoeff, cudaStream_t stream);
// valid_rows (device, may be NULL): rows at or past *valid_rows are skipped (tokens without an expert sit at
// the tail of pos[]; the dispatch kernel stores their start in offset[E]).
// CUDA-core GEMM: the LayerNorm output h, rows padded with zeros to padded_row(D) floats.
int launch_scatter_ln_rows(long long T, int D, const float* X, const float* score, const int* pos, const int* gate,
                           const float* gamma_all, const int* valid_rows, float* rscore, float* h, cudaStream_t stream);
// Tensor-core GEMM: packed FP16-pair plane `h` (pack_bytes) and two floats per row in row_info (token_row_info), of rows
// row0 .. row0 + T - 1.  gamma: the LayerNorm weights that launch_split_expert left for the first expert, or a copy of them,
// gamma_stride floats from one expert to the next.
int launch_scatter_ln_pack(long long row0, long long T, int D, const float* X, const float* score, const int* pos,
                           const int* gate, const float* gamma, size_t gamma_stride, const int* valid_rows, float* rscore,
                           void* h, float* row_info, cudaStream_t stream);
// launch_dispatch (without regions) and one of the two scatters in one kernel, where dispatch_scatter_supported.  gamma is
// what the scatter takes: with `pack` that of launch_split_expert, else the experts' LayerNorm weights.  early: the launch
// follows launch_route on this stream.
bool dispatch_scatter_supported(long long T, int D, int E, const float* X, bool pack);
int launch_dispatch_scatter(long long T, int D, int E, const float* X, const float* score, const int* gate,
                            const float* gamma, size_t gamma_stride, int* pos, int* count, int* offset, int* status,
                            int* zero, int zero_count, float* rscore, void* h, float* row_info, bool pack, bool early,
                            cudaStream_t stream);
int launch_gather(long long T, int D, const float* in, const int* pos, float* out, cudaStream_t stream,
                  const int* valid_rows = nullptr);
int launch_mix_gather(long long T, int D, const int* pos, const float* routed, const float* post,
                      const float* coeff, float* out, cudaStream_t stream, const int* valid_rows = nullptr);
int launch_layernorm(float* out, const float* in, long long n, int D, const float* gamma, cudaStream_t stream);
int launch_gelu_dot(const float* a, float* b, size_t len, cudaStream_t stream);
int launch_fill_int(int* dst, int value, cudaStream_t stream);   // *dst = value, stream ordered
// Tile-contiguous weight layouts (see rows.cu).
//   launch_retile        one matrix as raw FP32 tiles, for the CUDA-core GEMM (tiled_elems floats); src1 != NULL
//                        interleaves the rows of two matrices
//   launch_split_expert  both planes of an expert for the tensor-core GEMM (split_plane_elems floats each: FP16-pair
//                        tiles, 2^-s of every padded row, 32 words for the largest of the numbers behind them, one per
//                        neuron, column exponents, LayerNorm weights gamma' to use with the plane, see rows.cu)
int launch_retile(const float* src0, const float* src1, int M, int K, float* dst, cudaStream_t stream);
int launch_split_expert(const float* gamma, const float* wi0, const float* wi1, const float* wo, int D, int F, float* w01,
                        float* wo_dst, cudaStream_t stream);
inline size_t tiled_elems(int M, int K) { return (size_t)((M + 127) / 128) * 128 * (size_t)((K + 31) / 32) * 32; }
inline size_t split_range_at(int M, int K) { return tiled_elems(M, K) + (size_t)((M + 127) / 128) * 128; }
inline size_t split_columns_at(int M, int K) { return split_range_at(M, K) + 32 + (size_t)((M + 127) / 128) * 64; }
inline size_t split_gamma_at(int M, int K) { return split_columns_at(M, K) + (size_t)((K + 31) / 32) * 32; }
inline size_t split_plane_elems(int M, int K) { return split_gamma_at(M, K) + (size_t)((K + 31) / 32) * 32; }
// h = LN(x; gamma) for rows already in place, as launch_scatter_ln_rows / _pack write it (_pack: gamma' of the slot).
int launch_ln_rows(long long n, int D, const float* in, const float* gamma, float* h, cudaStream_t stream);
int launch_ln_pack(long long n, int D, const float* in, const float* gamma, void* h, float* row_info,
                   cudaStream_t stream);
// Bytes of an activation plane [rows][K], FP16 pairs or FP32 (rows padded to whole groups of 32 values).
inline size_t pack_bytes(long long rows, int K) { return (size_t)rows * (size_t)((K + 31) / 32) * 128; }

// CUDA-core GEMM.  Expert weights live in two raw FP32 planes in tile-contiguous layout (128 x 32 tiles):
// w01 [slots] x tiled(2F x D) (row 2f = wi_0[f], row 2f+1 = wi_1[f]) and wo [slots] x tiled(D x F).
// Activations h [T][padded_row(D)] and g [T][padded_row(F)] are FP32 (pack_bytes).
int launch_ffn_simt(long long T, int D, int F, int e_begin, int e_end, const int* offset, const int* slot_of_expert,
                    const float* h, const float* w01, const float* wo, float* g, const float* resid, float* out,
                    const int* out_pos, const float* mix_score, const unsigned long long* out_row_ptr, cudaStream_t stream);

// A one-warp kernel that waits, with the GEMM's bounded wait and the given limit, on a barrier nobody completes.
int launch_wait_probe(unsigned long long limit_ns, int* status, unsigned long long* waited_ns, cudaStream_t stream);

bool ffn_umma_supported(int D, int F, int E);
// Buffers of one tensor-core FFN call (all on the device).
struct FfnUmma {
    const int* offset;              // [E+1] first row of each expert
    bool early;                     // the launch follows launch_dispatch and launch_scatter_ln_pack, or, with `gate`,
    const int* gate;                // launch_dispatch_scatter on these gates: the first GEMM starts before the scatter ends
    const int* slot_of_expert;      // expert -> weight slot (NULL: identity)
    int slots;                      // weight slots in the planes
    const float *w01, *wo;          // split planes (launch_split_expert), [slots] x split_plane_elems
    const void* h;                  // packed LayerNorm output [T][D]
    const float* row_info;          // [T][2]
    void* g;                        // packed gate activations [T][F] (scratch)
    const float* resid;             // rows the experts were applied to
    // Output rows: row j of the experts' result goes to row out_pos[j] of `out` (out_pos NULL: row j), or to the
    // address out_row_ptr[out_pos[j]]; mix_score != NULL applies the base_layer output mix on the way.
    float* out;
    const int* out_pos;
    const float* mix_score;
    const unsigned long long* out_row_ptr;
    void* part;                     // scratch for cut tiles (ffn_umma_part_bytes; NULL: no tile is cut) and its
    size_t part_bytes;              // counters (FFN_COUNTERS, zero before the first launch of a call; every
    int* part_count;                // launch leaves them zero)
    int* status;
};
int launch_ffn_umma(const FfnUmma& f, long long T, int D, int F, int E, int e_begin, int e_end, int num_sms,
                    cudaStream_t stream, cudaEvent_t mid_event = nullptr);
constexpr int FFN_CTAS = 148;                   // most CTAs of a launch (SMs of a B200); the workspace is sized for them
constexpr int FFN_COUNTERS = FFN_CTAS * 16;      // ints in part_count: one per cut tile and accumulate warp
size_t ffn_umma_part_bytes(long long T, int D, int F);
// Rows of `in` [n][D] copied to the addresses dst[i] (one per row; they may point into a peer GPU's memory).
int launch_rows_to_ptrs(long long n, int D, const float* in, const unsigned long long* dst, cudaStream_t stream);

}  // namespace infmoe
