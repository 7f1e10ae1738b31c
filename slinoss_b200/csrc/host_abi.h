// Entry points of the library that only the package's own host module calls (not part of the C ABI): the decode step
// on strided operands and the small-batch linear layers around it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/slinoss_b200.h"

namespace sl {

// sl_v2x2ssd_fwd on the tensor-core path for 16-bit operands, that also leaves what a caller carries on from (in the operands'
// type): the end state (batch, heads, P, 2N), the last row of B (batch, groups, 2N) and of U (batch, heads, P).
// SL_ERR_UNSUPPORTED where another path would run; nothing is launched then.
struct ScanLast { void *state, *B, *U; };
SL_API int scan_fwd_last(const void* U, const float* M, const float* K, const void* B, const void* C, const float* initial_states,
                         const void* B_prev, const void* U_prev, void* Y, const ScanLast& last, int batch, int heads, int groups,
                         int T, int P, int N, int chunk, int io_dtype, int path, void* workspace, size_t workspace_bytes, void* stream);

struct MixerStepArgs {
  const void *gate, *value, *params, *bc;   // rows of the in_proj output, with their row strides (elements)
  int64_t gate_stride, value_stride, params_stride, bc_stride;
  const void *conv_weight, *conv_bias;
  void* conv_state;
  int d_conv;
  const float *dt_bias, *alpha_bias, *theta_mod_bias, *theta_bias, *theta_sign;
  const sl_scanprep_config* cfg;
  const float* d_skip;
  float* state;
  const void* b_prev_in;
  void* b_prev_out;   // may be b_prev_in when every head has its own group
  void* u_prev;
  void* workspace;    // receives the gated values (batch, heads * P) and their partial sums of squares
  size_t workspace_bytes;
  int batch, heads, groups, P, N, io_dtype;
  bool dependent = false;   // launched right behind a kernel of this library that wrote the rows
};

size_t mixer_step_workspace(int batch, int heads, int P);
// the partial sums of squares (batch, heads, 8) inside the workspace
inline float* step_partials(void* workspace, int batch, int heads, int P) {
  return reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + ((size_t)batch * heads * P * 4 + 255) / 256 * 256);
}
SL_API int mixer_step_launch(const MixerStepArgs& a, cudaStream_t st);
SL_API int mixer_step_norm(const void* workspace, const void* norm_weight, float eps, void* normed, int batch, int heads,
                           int P, int io_dtype, cudaStream_t st);

// y (M, O) = norm(x) W^T + bias, 16-bit, M <= 64 rows.  norm: none, or RMSNorm whose sums of squares are given as partials
// per row.
struct SkinnyArgs {
  const void* x;          // (M, K), row stride x_stride
  int64_t x_stride;
  const void* norm_weight;   // (K) or null
  float norm_eps;
  const float* partials;  // (M, n_partials), with norm_weight
  int n_partials;
  const void *weight, *bias;   // (O, K) dense, bias (O) or null
  void* out;              // (M, O) dense
  int M, K, O, io_dtype;
  bool dependent = false;   // launched right behind a kernel of this library that wrote x (and no parameter)
};
SL_API bool skinny_supported(int M, int K, int O, int io_dtype);
SL_API int skinny_linear(const SkinnyArgs& a, cudaStream_t st);

// One linear layer of a block's token and what follows it (token_linear.cu): x (M, K) dense, weight (O, K) dense, M <= 64.
struct TokenLinearArgs {
  const void *x, *weight, *bias;   // bias (O) or null
  void* out[3];                    // dense (M, width[i]) each, the columns in turn; swiglu: one of O / 2
  int width[3];
  const void* residual;            // (M, O) or null: added to the rounded product
  int M, K, O, io_dtype;
  bool gelu, swiglu;               // activation of the rounded product; swiglu: value rows, then gate rows
  // of x first, M <= 16: RMSNorm with the bits of sl_rmsnorm_fwd, or with the partial sums of squares of mixer_step_norm
  const void* norm_weight = nullptr;
  float norm_eps = 0.f;
  const float* partials = nullptr;
  int n_partials = 0;
  bool dependent = false;          // launched right behind a kernel of this library (which writes no parameter)
};
SL_API bool token_linear_supported(const TokenLinearArgs& a);
SL_API int token_linear(const TokenLinearArgs& a, cudaStream_t st);

// ---- scan preparation and mixer tail on strided rows ---------------------------------------------------------------------
// Operands and results are rows of (batch * T) with a row stride each (columns of the in_proj output and of its
// gradient); a null pointer skips its part, as in sl_scanprep_conv_fwd / _bwd.
struct ScanPrepArgs {
  const void* value; int64_t value_stride;
  const void *conv_weight, *conv_bias, *conv_state_in;
  void* conv_state_out;
  int d_conv;
  const void* params; int64_t params_stride;
  const void* bc; int64_t bc_stride;
  const float *dt_bias, *alpha_bias, *theta_mod_bias, *theta_bias, *theta_sign;
  const sl_scanprep_config* cfg;
  int64_t u_b, u_h, u_t;                    // strides of U (dU)
  int batch, heads, groups, T, P, N, io_dtype;
};
struct ScanPrepOut { void* U; float *M, *K; void *B, *C; };
struct ScanPrepGrads {
  const void* dU; const float *dM, *dK; const void *dB, *dC;
  void* d_value; int64_t d_value_stride;
  float *d_conv_weight, *d_conv_bias;
  void* d_conv_state;
  void* d_params; int64_t d_params_stride;
  void* d_bc; int64_t d_bc_stride;
  float *d_dt_bias, *d_alpha_bias, *d_theta_mod_bias, *d_theta_bias;
  const void* dY = nullptr;       // with skip: the gradient of U is dU + skip[head] * dY (dY laid out like dU)
  const float* skip = nullptr;
};
SL_API int scanprep_fwd(const ScanPrepArgs& a, const ScanPrepOut& o, cudaStream_t st);
SL_API int scanprep_bwd(const ScanPrepArgs& a, const ScanPrepGrads& g, cudaStream_t st);
SL_API int mixer_tail_bwd(const void* Y, const void* gate, int64_t gate_stride, const void* skip, const float* d_skip,
                          const void* norm_weight, float eps, const void* d_normed, void* dY, void* d_gate,
                          int64_t d_gate_stride, void* d_skip_input, float* d_d_skip, float* d_norm_weight, int batch, int heads,
                          int T, int P, int io_dtype, cudaStream_t st);

// ---- row kernels whose sums over rows do not depend on the schedule -----------------------------------------------------
// d_weight float32 or weight64 (sums that rounding to a shorter type makes independent of their order): added to; extra
// (rows, C) or null is added to d_x, and its column sums to extra_sum (or null) where rmsnorm_bwd_sums_extra
SL_API bool rmsnorm_bwd_sums_extra(int C);
SL_API int rmsnorm_bwd(const void* x, const void* weight, float eps, const void* d_out, const void* extra, void* d_x, float* d_weight,
                       double* weight64, double* extra_sum, long long rows, int C, int io_dtype, cudaStream_t st);
// out = a + b of n elements, rounded as torch rounds the sum of two such tensors
SL_API int residual_sum(const void* a, const void* b, void* out, long long n, int io_dtype, cudaStream_t st);
// sl_ffn_activation_bwd that also adds the column sums of its result to sums (one or two times H)
SL_API int ffn_act_bwd_sum(const void* projected, const void* d_hidden, void* d_projected, double* sums, long long rows, int H, int kind,
                           int io_dtype, cudaStream_t st);
SL_API size_t column_sum_partials(long long rows, int C, int io_dtype);
SL_API int column_sum(const void* x, void* out, float* partial, long long rows, int C, int io_dtype, cudaStream_t st);

// ---- language-model training step ------------------------------------------------------------------------------------
SL_API int cross_entropy_fwd(const void* logits, const int64_t* target, float* loss, float* lse, int64_t rows, int V, int io,
                             cudaStream_t st);
SL_API int cross_entropy_finish(const float* loss, const int64_t* target, int64_t rows, bool mean, float* total, float* scale,
                                cudaStream_t st);
SL_API int cross_entropy_bwd(const void* logits, const int64_t* target, const float* lse, const float* g, const float* scale, void* d,
                             int64_t rows, int V, int io, cudaStream_t st);
// ids sorted (stable) and the positions they came from -> dE (V, C)
SL_API int embedding_bwd(const int* sorted, const int64_t* order, const void* d_out, void* dE, int n, int V, int C, int io,
                         cudaStream_t st);
// lists of tensors by value; first[i] = chunks of the tensors before i
constexpr int MT_MAX = 72;
struct MtList1 { const void* p[MT_MAX]; int64_t len[MT_MAX]; unsigned first[MT_MAX]; int n; };
struct MtList4 { void *p[MT_MAX], *g[MT_MAX], *m[MT_MAX], *v[MT_MAX]; int64_t len[MT_MAX]; unsigned first[MT_MAX]; int n; };
// what beta does not hold to float32 precision near one is formed in float64: 1 - beta, ln beta, 1 - lr * weight_decay
struct AdamWArgs { float lr, eps, decay, beta2, one_minus_beta1, one_minus_beta2; double ln_beta1, ln_beta2; const float *step, *grad_scale; };
SL_API unsigned mt_chunks(int64_t len);
SL_API int multi_sumsq(const MtList1& list, unsigned chunks, float* partial, int io, cudaStream_t st);
SL_API int norm_finish(const float* partial, int n, float clip, float* out, cudaStream_t st);
SL_API int multi_adamw(const MtList4& list, unsigned chunks, const AdamWArgs& a, int io, cudaStream_t st);

}  // namespace sl
