// Internal launcher declarations shared by the kernel translation units and the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nvfp4_b200.h"

namespace nvfp4 {

// quant_kernels.cu --------------------------------------------------------------------------
int launch_row_amax(cudaStream_t s, const void* x, int dtype, float* out, uint32_t rows, uint32_t row_len);
// partials (optional, kAmaxPartials floats): every CTA leaves its maximum there -- tensor_amax_partials(n) of them -- for
// a consumer that reduces them, and `out` is not touched (no zeroing launch, no atomics).
constexpr uint32_t kAmaxPartials = 148u * 4u;
// max_partials: more of them where the buffer holds a float per 1024 values (chunk scratch): twice the loads in flight, 524 MB of
// bf16 80 us instead of 91.
constexpr uint32_t kAmaxScratchPartials = 148u * 8u;
uint32_t tensor_amax_partials(uint64_t n, uint32_t max_partials = kAmaxPartials);
int launch_tensor_amax(cudaStream_t s, const void* x, int dtype, float* chunk_amax, float* out, uint64_t n,
                       float* partials = nullptr, uint32_t max_partials = kAmaxPartials);
// partials (optional): kAmaxScratchPartials floats, as above.  out_cleared: out[0] is not cleared first, its value takes part
int launch_nvfp4_amax(cudaStream_t s, const uint8_t* bytes, const uint8_t* scales, const float* gscales, uint32_t rows,
                      uint32_t cols, int rowwise, int packed, float* chunk_amax, float* out, float* partials = nullptr,
                      bool out_cleared = false);
// transform 0: out[0] = max(chunks); 1: out[0] = MS-EDEN global scale of that max
int launch_amax_from_chunks(cudaStream_t s, const float* chunk_amax, float* out, uint32_t chunk_count, int transform);
int launch_ms_eden_scale_from_amax(cudaStream_t s, const float* amax, float* out);
// relu2: quantize relu(x)^2 computed on load; decoded_amax (optional f32[1]): max |decoded value| of the result, cleared first
// unless decoded_cleared
int launch_four_six(cudaStream_t s, const void* x, int dtype, const float* amax, int rowwise, uint32_t rows,
                    uint32_t cols, uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs, int relu2 = 0,
                    float* decoded_amax = nullptr, uint32_t amax_count = 1, bool decoded_cleared = false);
int launch_four_six_rowwise_fused(cudaStream_t s, const void* x, int dtype, uint32_t rows, uint32_t cols,
                                  uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs, float* out_amax,
                                  float* decoded_amax, int relu2 = 0, bool decoded_cleared = false);
int launch_four_six_padded(cudaStream_t s, const float* x, const float* amax, uint8_t* out_fp4, uint8_t* out_scales,
                           float* out_gs, uint32_t rows, uint32_t cols, uint32_t padded_rows, uint32_t padded_cols,
                           int transposed);
int launch_packed_scale_pad(cudaStream_t s, uint8_t* packed, uint32_t rows, uint32_t k_dim);
// y = z + beta * (x - z) -> tensor amax -> four-six (tensor scale); chunk_amax optional
int launch_schedule_free_materialize(cudaStream_t s, const float* z, const float* x, float beta, float* chunk_amax,
                                     float* amax, uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs,
                                     uint32_t rows, uint32_t cols, float* partials = nullptr);
// amax_in / gs_out (optional): the global scale is the MS-EDEN scale of max(0, amax_in[0 .. amax_count - 1]), or of amax_in[0]
// as it stands for a count of 0 (derived inside the kernel where the kernel supports it, by a one-thread kernel otherwise),
// and is written to gs_out[0]; a.global_scale and a.host_global_scale are then not read.  amax_count > 0 only where
// ms_eden_takes_amax.
int launch_ms_eden(cudaStream_t s, const nvfp4_ms_eden_args& a, const float* amax_in = nullptr, float* gs_out = nullptr,
                   uint32_t amax_count = 0);
bool ms_eden_takes_amax(const nvfp4_ms_eden_args& a);
// Pair quantization; when col_sum_partials != nullptr (and ms_eden_pair_is_tiled) it also writes the
// per-row-tile column sums [ms_eden_pair_row_tiles(rows)][cols] for launch_col_sum_reduce.
// amax_in / gs_out (only when ms_eden_pair_takes_amax): the kernel derives the global scale from the same maximum
// itself and writes it to gs_out[0]; rows.global_scale / transposed.global_scale are then not read.
// beside_others: kernels of another stream are waiting for room on the SMs that this one would take by starting early.
// zero (likewise only when ms_eden_pair_takes_amax): zero_words 16-byte words that the kernel clears beside its work.
int launch_ms_eden_pair(cudaStream_t s, const nvfp4_ms_eden_args& rows, const nvfp4_ms_eden_args& transposed,
                        float* col_sum_partials = nullptr, const float* amax_in = nullptr, float* gs_out = nullptr,
                        uint32_t amax_count = 0, void* zero = nullptr, uint64_t zero_words = 0, bool beside_others = false);
bool ms_eden_pair_takes_amax(const nvfp4_ms_eden_args& rows, const nvfp4_ms_eden_args& transposed);
bool ms_eden_pair_is_tiled(const nvfp4_ms_eden_args& rows, const nvfp4_ms_eden_args& transposed);
uint32_t ms_eden_pair_row_tiles(uint32_t rows);
int launch_col_sum_reduce(cudaStream_t s, const float* partials, float* dbias, uint32_t tiles, uint32_t n);
int launch_decode(cudaStream_t s, const uint8_t* bytes, const uint8_t* scales, const float* gscales, int rowwise,
                  int transpose, float* out, uint32_t rows, uint32_t cols);
int launch_scale_pack(cudaStream_t s, const uint8_t* logical, uint8_t* packed, uint32_t mn, uint32_t k_dim);
// two planes of one k_dim (the operands of a GEMM), in one launch where both allow the tiled kernel
int launch_scale_pack_pair(cudaStream_t s, const uint8_t* const (&logical)[2], uint8_t* const (&packed)[2],
                           const uint32_t (&mn)[2], uint32_t k_dim);
int launch_pad_u4_rows(cudaStream_t s, const uint8_t* src, uint8_t* dst, uint32_t rows, uint32_t padded_rows,
                       uint32_t cols);
int launch_pad_f32(cudaStream_t s, const float* src, float* dst, uint32_t rows, uint32_t cols, uint32_t padded_rows,
                   uint32_t padded_cols, int transpose);
int launch_crop_f32(cudaStream_t s, const float* src, float* dst, uint32_t rows, uint32_t src_cols, uint32_t dst_cols);
int launch_postop(cudaStream_t s, float* raw, float* other, const uint8_t* bias_bytes, const uint8_t* bias_scales,
                  const float* bias_gs, uint32_t rows, uint32_t cols, int mode);
int launch_bias_grad(cudaStream_t s, const void* e, int dtype, float* dbias, uint32_t tokens, uint32_t n);
// d_pre = (d_out * 2) * max(pre, 0); pre_kind 0 f32, 1 bf16, 2 f16; gradients f32 or (grad_bf16) bf16.
// chunk_amax (optional, relu2_backward_grid(n) floats): per-CTA amax of the stored gradient.
int launch_relu2_backward(cudaStream_t s, const void* pre, int pre_kind, const void* d_out, void* d_pre, int grad_bf16,
                          uint64_t n, float* chunk_amax = nullptr);
uint32_t relu2_backward_grid(uint64_t n);

// gemm_tcgen05.cu ---------------------------------------------------------------------------
// Two GEMMs of a stream that need nothing of one another run side by side where the first is launched with kLetsNextBeside and the
// second, directly behind it, with kBesidePrior: the second starts on the SMs that the first leaves, and ends behind it, so that
// what follows is ordered behind both.  The second's memory must lie apart from what the first reads and writes.  dX and dW of a
// linear: neither grid fills the SMs evenly, and the second's set-up and fill run beside the first's last wave: backward of
// 1000 x 3072 f32 41.9 -> 39.6 us, 512 x 768 bf16 28.3 -> 23.2, 8192 x 2304 76.9 -> 75.5.  On the side stream instead, behind an
// event of its own, dW took 43.5 in the first and 75.8 in the last.
enum class GemmNeighbour { kNone, kLetsNextBeside, kBesidePrior };
// out_is_zero: the output holds zeros already (it is cleared first where gemm_adds_into_output otherwise)
// row_amax_cleared: so does a.relu2_row_amax
// neighbour: the role asked for; launched_as: the one taken.  A GEMM that is timed, or would run beside its predecessor but clears
// its output itself, takes none.
int launch_gemm(cudaStream_t s, const nvfp4_gemm_args& a, bool out_is_zero = false, bool row_amax_cleared = false,
                GemmNeighbour neighbour = GemmNeighbour::kNone, GemmNeighbour* launched_as = nullptr);
// Whether launch_gemm splits K and sums the partial tiles in the output.
bool gemm_adds_into_output(const nvfp4_gemm_args& a);
// What launch_gemm would choose for these arguments on the current device (no launch).
int gemm_plan_query(const nvfp4_gemm_args& a, nvfp4_gemm_plan* out, uint32_t* pair);
// Encodes (and keeps in the calling thread's cache) the operand tensor maps of a GEMM ahead of its launch.
int gemm_prepare_operand_maps(const uint8_t* a_bytes, const uint8_t* b_bytes, uint32_t m, uint32_t k, uint32_t n);
// Measurement / test aids: forced tile shape (block_n 0 = automatic), limit of the kernel's bounded waits,
// debug flags (bit 0: CTA 0 of every GEMM never loads its first k-tile), tensor-map cache counters.
void gemm_set_tile_override(int block_m, int block_n);
void gemm_set_wait_timeout_ns(uint64_t ns);
void gemm_set_debug_flags(uint32_t flags);
void gemm_map_cache_stats(uint64_t* hits, uint64_t* misses);
// 1: split-K never uses more than two splits (run-to-run identical sums); 0 (default): as many as fill the SMs
void gemm_set_deterministic(int on);
int gemm_get_deterministic();
int gemm_timing_begin(uint32_t max_records);
int gemm_timing_end(uint32_t* count, double* total_ms, double* total_flops, float* per_launch_ms,
                    double* per_launch_flops, uint32_t capacity);
// Device status word written by kernels whose bounded waits expired (0 = never).
uint32_t* device_status_word();

void set_last_error(const char* msg);
// Host-side tally of kernel launches made by this library (read through nvfp4_launch_count).
void count_launch();

// Launches a kernel that may start while the kernel before it in the stream drains (programmatic stream serialization).
// Only for kernels whose every thread waits for that one before its first access to memory
// (wait_for_prior_then_allow_next): launch latency and the start of the thread blocks then cost nothing behind another
// kernel.  The main path's kernels are; those for shapes and alignments that it does not take (ms_eden_kernel,
// ms_eden_tile_kernel, four_six_padded_kernel, decode_kernel, scale_pack_kernel, packed_scale_pad_kernel, bias_grad_kernel) and
// relu2_backward_kernel are launched plainly: their loads are not pinned behind the wait.
template <typename... Params, typename... Args>
int launch_chained(void (*kernel)(Params...), dim3 grid, uint32_t threads, size_t shared_bytes, cudaStream_t s, const Args&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = shared_bytes;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t launched = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  count_launch();
  const cudaError_t last = cudaGetLastError();
  return static_cast<int>(launched != cudaSuccess ? launched : last);
}

}  // namespace nvfp4
