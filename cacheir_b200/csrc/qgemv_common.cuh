// Arguments shared by the dequant-GEMV kernels and their launchers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cb200 {

// Fused QKV epilogue: RoPE on the q and k heads, new k/v rows written into the page pool.
struct RopeAppendParams {
  const float* table;          // [table_positions][head_dim/2] (cos, sin) pairs, or null: evaluate on the fly
  int table_positions;
  const int32_t* positions;    // [M] position of the token of each batch row
  const int32_t* page_table;   // [M][max_pages]
  void* k_cache;               // [slots][kv_heads][page_size][head_dim], fp16
  void* v_cache;
  int q_dim, k_dim, head_dim, kv_heads, max_pages, page_size;
  float theta;
};
constexpr int kEpiQkvRopeAppend = 3;   // internal epilogue code (cacheir_b200_qkv_rope_append)

struct QGemvParams {
  const void* x;
  const void* packed;
  const void* scales;
  const float* zero_points;
  const void* residual;
  void* y;
  int M, N, K;
  int bits;        // 8, 4, or 0 for dense weights of x's type
  int group_size;  // 0: one (scale, zero) per row; >0: symmetric groups along K
  int x_dtype, scale_dtype;
  long long x_stride;
  int epilogue;
  bool vector_ok;  // rows of x and of the packed weight can be read in 16-byte units
  bool tiled;      // codes are in the 128x128 tile order of cacheir_b200_pack_relayout
  bool paired;     // tiled, and every tile pairs 64 rows of the first half of W with the matching 64 of the second half
  bool x_prequantized;  // the workspace already holds the integer form of x (see cacheir_b200_quantize_activations)
  const void* norm_weight;  // non-null: y = epilogue(rmsnorm(x; norm_weight, norm_eps) . W^T): the norm runs inside the activation pre-pass (integer tensor-core path only)
  float norm_eps;
  RopeAppendParams rope;  // epilogue == kEpiQkvRopeAppend only
};

int launch_qgemv_cuda_core(const QGemvParams& p, cudaStream_t stream);
// Streaming int4 GEMV for up to 8 batch rows (mma.sync on nibbles unpacked in registers, row-major codes).
bool qgemv_mma_supported(const QGemvParams& p);
int launch_qgemv_mma(const QGemvParams& p, cudaStream_t stream);

// Streaming dequant-GEMV for up to 32 rows (warp MMAs on codes unpacked in registers; both code layouts).
bool qgemv_stream_supported(const QGemvParams& p);
int launch_qgemv_stream(const QGemvParams& p, cudaStream_t stream);
int qgemv_stream_plan(const QGemvParams& p);   // (row groups << 4) | CTAs along K that the launcher would choose

// int4 dequant-GEMM for up to 128 rows with the weights in tensor memory (both code layouts).
bool qgemm_w4_supported(const QGemvParams& p);
bool qgemm_w4_preferred(const QGemvParams& p);  // is it the fastest of the int4 products?
int launch_qgemm_w4(const QGemvParams& p, cudaStream_t stream);
int qgemm_w4_plan(const QGemvParams& p);        // 128 | (4 << 4) | CTAs along K
int qgemm_w4_device_status(bool reset);

// Tensor-core (tcgen05) small-M GEMM: weights are the 128-row MMA operand.
bool qgemm_tc_supported(const QGemvParams& p);
int launch_qgemm_tc(const QGemvParams& p, cudaStream_t stream);
// Integer tensor-core path (int8 per-row weights, fp16 activations turned into 16-bit fixed point).
// Needs `qgemm_i8_workspace_bytes` of caller scratch for the activation bytes.
size_t qgemm_i8_workspace_bytes(int M, int K);
bool qgemm_i8_supported(const QGemvParams& p, const void* workspace, size_t workspace_bytes);
int launch_qgemm_i8(const QGemvParams& p, void* workspace, cudaStream_t stream);
int qgemm_i8_plan(const QGemvParams& p);   // the split-K factor the launcher would use
int qgemm_i8_device_status(bool reset);
int qgemv_mma_device_status(bool reset);
int qgemm_i8_quantize_activations(const void* x, long long x_stride, int M, int K, void* workspace, cudaStream_t stream);
int qgemm_i8_rms_norm_quantize(const void* x, const void* residual, const void* weight, void* sum_out, void* out, int M,
                               int hidden, float eps, void* workspace, cudaStream_t stream);
// Prompts and other batches of more than 64 rows on the integer tensor cores (qgemm_i8_rows.cu): blocks of 128 rows.
// `n_rows` (device, may be null): only the first *n_rows of the M rows are real.
struct TallPlanes {
  int8_t* planes;   // [row block][k block][128 high, 128 low rows][128 bytes]
  float* sx;
  int* qsum;
};
TallPlanes tall_planes(void* workspace, int M, int K);
int qgemm_i8_quantize_tall(const void* x, long long x_stride, int M, const int* n_rows, int K, void* workspace, cudaStream_t stream);
int qgemm_i8_rms_norm_quantize_tall(const void* x, const void* weight, int M, const int* n_rows, int hidden, float eps, void* workspace,
                                    cudaStream_t stream);
bool qgemm_i8_rows_supported(const QGemvParams& p, const void* workspace, size_t workspace_bytes);
// Is that faster than passes of 64 rows?
bool qgemm_i8_rows_preferred(const QGemvParams& p);
int launch_qgemm_i8_rows(const QGemvParams& p, const int* n_rows, void* workspace, cudaStream_t stream);
int qgemm_i8_rows_device_status(bool reset);
// Device-side status word of the tensor-core kernel (0 = no bounded wait ever gave up).
int qgemm_tc_device_status(bool reset);

}  // namespace cb200
