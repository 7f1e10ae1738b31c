// Kernels of the language-model training step around the stack: cross-entropy over the vocabulary, the gradient of the
// token embedding, the global gradient norm and AdamW.  All are bound by HBM traffic (or, for the narrow models, by
// launches): each reads and writes what it must once, in 16-byte pieces.
#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

constexpr int64_t CE_IGNORE = -100;   // the target that torch's cross-entropy leaves out by default

template <bool PRECISE> __device__ __forceinline__ float exp_io(float x) { return PRECISE ? expf(x) : __expf(x); }

// ---- cross-entropy -------------------------------------------------------------------------------------------------
// One CTA per row of logits, read once with an online maximum (the library route made a float32 copy of the logits,
// a second float32 tensor of log-probabilities and, backwards, two more: about 14 bytes per logit each way; here 2
// forward and 4 backward.  16380 x 32000 bf16, forward + backward: 4.4 -> 0.6 ms).
template <typename T, bool VEC>
__global__ void __launch_bounds__(512) ce_fwd_kernel(const T* __restrict__ logits, const int64_t* __restrict__ target,
                                                     float* __restrict__ loss, float* __restrict__ lse, int V) {
  constexpr int W = VEC ? Vec16<T>::N : 1;
  constexpr bool PRECISE = sizeof(T) == 4;
  __shared__ float s_m[16], s_s[16];
  const size_t row = blockIdx.x;
  const T* x = logits + row * V;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float m = -INFINITY, s = 0.f;
  for (int c = threadIdx.x; c < V / W; c += blockDim.x) {
    float v[W];
    if constexpr (VEC) load16<T>(x + (size_t)c * W, v); else v[0] = to_f32(x[c]);
    float mx = v[0];
#pragma unroll
    for (int k = 1; k < W; ++k) mx = fmaxf(mx, v[k]);
    if (mx > m) { s *= exp_io<PRECISE>(m - mx); m = mx; }
    if (m == -INFINITY) continue;
#pragma unroll
    for (int k = 0; k < W; ++k) s += exp_io<PRECISE>(v[k] - m);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o), mm = fmaxf(m, m2);
    s = mm == -INFINITY ? 0.f : s * exp_io<PRECISE>(m - mm) + s2 * exp_io<PRECISE>(m2 - mm);
    m = mm;
  }
  if (lane == 0) { s_m[w] = m; s_s[w] = s; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mm = s_m[0];
    for (int k = 1; k < nw; ++k) mm = fmaxf(mm, s_m[k]);
    float tot = 0.f;
    for (int k = 0; k < nw; ++k) tot += s_m[k] == -INFINITY ? 0.f : s_s[k] * exp_io<PRECISE>(s_m[k] - mm);
    const float l = mm + logf(tot);
    const int64_t t = target[row];
    lse[row] = l;
    loss[row] = t >= 0 && t < V ? l - to_f32(x[t]) : t == CE_IGNORE ? 0.f : NAN;
  }
}

// total: the rows' losses summed in float64 times scale, the reciprocal of the number of rows that are not
// ignored, or one
__global__ void __launch_bounds__(1024) ce_finish_kernel(const float* __restrict__ loss, const int64_t* __restrict__ target,
                                                         int64_t rows, bool mean, float* __restrict__ total,
                                                         float* __restrict__ scale_out) {
  __shared__ double s_sum[32];
  __shared__ int s_n[32];
  double sum = 0.0;
  int n = 0;
  for (int64_t i = threadIdx.x; i < rows; i += 1024) { sum += loss[i]; n += target[i] != CE_IGNORE; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); n += __shfl_xor_sync(0xffffffffu, n, o); }
  if ((threadIdx.x & 31) == 0) { s_sum[threadIdx.x >> 5] = sum; s_n[threadIdx.x >> 5] = n; }
  __syncthreads();
  if (threadIdx.x == 0) {
    sum = 0.0; n = 0;
    for (int k = 0; k < 32; ++k) { sum += s_sum[k]; n += s_n[k]; }
    const double scale = mean ? 1.0 / n : 1.0;
    total[0] = (float)(sum * scale);    // (every row ignored: 0 / 0)
    scale_out[0] = (float)scale;
  }
}

// d logits = (softmax - onehot) * g * scale, both device scalars; zeros in ignored rows
template <typename T, bool VEC>
__global__ void __launch_bounds__(512) ce_bwd_kernel(const T* __restrict__ logits, const int64_t* __restrict__ target,
                                                     const float* __restrict__ lse, const float* __restrict__ g,
                                                     const float* __restrict__ scale, T* __restrict__ d, int V) {
  constexpr int W = VEC ? Vec16<T>::N : 1;
  constexpr bool PRECISE = sizeof(T) == 4;
  const size_t row = blockIdx.x;
  const T* x = logits + row * V;
  T* o = d + row * V;
  const int64_t t = target[row];
  if (t == CE_IGNORE) {
    const float zero[W] = {};
    for (int c = threadIdx.x; c < V / W; c += blockDim.x) {
      if constexpr (VEC) store16<T>(o + (size_t)c * W, zero); else o[c] = from_f32<T>(0.f);
    }
    return;
  }
  const float l = lse[row], f = g[0] * scale[0];
#pragma unroll 2
  for (int c = threadIdx.x; c < V / W; c += blockDim.x) {
    float v[W];
    if constexpr (VEC) load16<T>(x + (size_t)c * W, v); else v[0] = to_f32(x[c]);
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] = (exp_io<PRECISE>(v[k] - l) - (c * W + k == t ? 1.f : 0.f)) * f;
    if constexpr (VEC) store16<T>(o + (size_t)c * W, v); else o[c] = from_f32<T>(v[0]);
  }
}

// ---- embedding gradient ----------------------------------------------------------------------------------------------
// dE[v] = sum of d_out over the positions of token v, in float32, in position order.  One CTA per vocabulary row finds
// its run in the sorted ids by bisection and writes its row once (zeros where the token does not occur: no memset).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) embedding_bwd_kernel(const int* __restrict__ sorted, const int64_t* __restrict__ order,
                                                            const T* __restrict__ d_out, T* __restrict__ dE, int n, int C) {
  constexpr int W = VEC ? Vec16<T>::N : 1;
  const int v = blockIdx.x;
  auto lower = [&](int key) {
    int lo = 0, hi = n;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (sorted[mid] < key) lo = mid + 1; else hi = mid; }
    return lo;
  };
  const int a = lower(v), b = lower(v + 1);
  for (int c = threadIdx.x; c < C / W; c += blockDim.x) {
    float acc[W];
#pragma unroll
    for (int k = 0; k < W; ++k) acc[k] = 0.f;
#pragma unroll 4
    for (int i = a; i < b; ++i) {
      float x[W];
      const T* src = d_out + (size_t)order[i] * C + (size_t)c * W;
      if constexpr (VEC) load16<T>(src, x); else x[0] = to_f32(*src);
#pragma unroll
      for (int k = 0; k < W; ++k) acc[k] += x[k];
    }
    if constexpr (VEC) store16<T>(dE + (size_t)v * C + (size_t)c * W, acc); else dE[(size_t)v * C + c] = from_f32<T>(acc[0]);
  }
}

// ---- multi-tensor kernels ---------------------------------------------------------------------------------------------
// A CTA owns one chunk of MT_CHUNK elements of one tensor of the list; the list travels in the kernel's parameters.
constexpr int MT_CHUNK = 256 * 8 * 4;
template <typename S>
__device__ __forceinline__ int find_tensor(const S& list, unsigned chunk) {
  int lo = 0, hi = list.n - 1;
  while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (list.first[mid] <= chunk) lo = mid; else hi = mid - 1; }
  return lo;
}

template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(MtList1 list, float* __restrict__ partial) {
  constexpr int W = Vec16<T>::N;
  __shared__ float s_red[8];
  const int ti = find_tensor(list, blockIdx.x);
  const T* x = reinterpret_cast<const T*>(list.p[ti]);
  const size_t base = (size_t)(blockIdx.x - list.first[ti]) * MT_CHUNK, end = min((size_t)list.len[ti], base + MT_CHUNK);
  float ss = 0.f;
  if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
#pragma unroll 4
    for (size_t i = base + threadIdx.x * W; i + W <= end; i += 256 * W) {
      float v[W];
      load16<T>(x + i, v);
#pragma unroll
      for (int k = 0; k < W; ++k) ss += v[k] * v[k];
    }
    for (size_t i = base + (end - base) / W * W + threadIdx.x; i < end; i += 256) { const float v = to_f32(x[i]); ss += v * v; }
  } else {
    for (size_t i = base + threadIdx.x; i < end; i += 256) { const float v = to_f32(x[i]); ss += v * v; }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) tot += s_red[k];
    partial[blockIdx.x] = tot;
  }
}
// norm = sqrt(sum of partials); scale = max(1, (norm + 1e-6) / clip)
__global__ void __launch_bounds__(1024) norm_finish_kernel(const float* __restrict__ partial, int n, float clip,
                                                           float* __restrict__ out) {
  __shared__ double s_red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 1024) s += partial[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int k = 0; k < 32; ++k) tot += s_red[k];
    const float norm = (float)sqrt(tot);
    out[0] = norm;
    out[1] = fmaxf((norm + 1e-6f) / clip, 1.f);
  }
}

// AdamW with decoupled decay; states in the parameter's type, arithmetic in float32.  A gradient scale other than one
// divides the gradients as they are read and is written back to them.
template <typename T>
__global__ void __launch_bounds__(256) adamw_kernel(MtList4 list, AdamWArgs a) {
  constexpr int W = Vec16<T>::N;
  const int ti = find_tensor(list, blockIdx.x);
  T* p = reinterpret_cast<T*>(list.p[ti]);
  T* g = reinterpret_cast<T*>(list.g[ti]);
  T* m = reinterpret_cast<T*>(list.m[ti]);
  T* v = reinterpret_cast<T*>(list.v[ti]);
  const size_t base = (size_t)(blockIdx.x - list.first[ti]) * MT_CHUNK, end = min((size_t)list.len[ti], base + MT_CHUNK);
  const float step = a.step[0], gs = a.grad_scale ? a.grad_scale[0] : 1.f;
  // bias corrections 1 - beta^step = -(e^(step ln beta) - 1): the product in float64, so that they keep float32 precision
  // for beta near one (1 - 0.999 in float32 is off by 5e-5)
  const float bc1 = -expm1f((float)(step * a.ln_beta1)), bc2s = sqrtf(-expm1f((float)(step * a.ln_beta2)));
  const float step_size = a.lr / bc1;
  auto update = [&](float& pv, float& gv, float& mv, float& vv) {
    gv = gs == 1.f ? gv : gv / gs;
    pv *= a.decay;
    mv += a.one_minus_beta1 * (gv - mv);
    vv = a.beta2 * vv + a.one_minus_beta2 * gv * gv;
    pv -= step_size * mv / (sqrtf(vv) / bc2s + a.eps);
  };
  const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
                     reinterpret_cast<uintptr_t>(v)) & 15) == 0;
  size_t tail = base;
  if (vec) {
    tail = base + (end - base) / W * W;
#pragma unroll 2
    for (size_t i = base + threadIdx.x * W; i < tail; i += 256 * W) {
      float pv[W], gv[W], mv[W], vv[W];
      load16<T>(p + i, pv); load16<T>(g + i, gv); load16<T>(m + i, mv); load16<T>(v + i, vv);
#pragma unroll
      for (int k = 0; k < W; ++k) update(pv[k], gv[k], mv[k], vv[k]);
      store16<T>(p + i, pv); store16<T>(m + i, mv); store16<T>(v + i, vv);
      if (gs != 1.f) store16<T>(g + i, gv);
    }
  }
  for (size_t i = tail + threadIdx.x; i < end; i += 256) {
    float pv = to_f32(p[i]), gv = to_f32(g[i]), mv = to_f32(m[i]), vv = to_f32(v[i]);
    update(pv, gv, mv, vv);
    p[i] = from_f32<T>(pv); m[i] = from_f32<T>(mv); v[i] = from_f32<T>(vv);
    if (gs != 1.f) g[i] = from_f32<T>(gv);
  }
}

inline int row_threads(int pieces) { return pieces >= 2048 ? 512 : pieces >= 128 ? 256 : 128; }

}  // namespace

#define SL_VEC_DISPATCH(ok, ...)            \
  do {                                      \
    if (ok) { constexpr bool VEC = true; __VA_ARGS__; } \
    else { constexpr bool VEC = false; __VA_ARGS__; }   \
  } while (0)

int cross_entropy_fwd(const void* logits, const int64_t* target, float* loss, float* lse, int64_t rows, int V, int io,
                      cudaStream_t st) {
  if (rows < 1 || V < 1) return SL_ERR_BAD_SHAPE;
  const int w = io == SL_F32 ? 4 : 8;
  SL_DISPATCH_DTYPE(io, T, SL_VEC_DISPATCH(V % w == 0 && aligned(logits, 16), {
    ce_fwd_kernel<T, VEC><<<(unsigned)rows, row_threads(V / w), 0, st>>>(reinterpret_cast<const T*>(logits), target, loss, lse, V);
  }));
  note_launches(1);
  return launch_status();
}
int cross_entropy_finish(const float* loss, const int64_t* target, int64_t rows, bool mean, float* total, float* scale,
                         cudaStream_t st) {
  ce_finish_kernel<<<1, 1024, 0, st>>>(loss, target, rows, mean, total, scale);
  note_launches(1);
  return launch_status();
}
int cross_entropy_bwd(const void* logits, const int64_t* target, const float* lse, const float* g, const float* scale, void* d,
                      int64_t rows, int V, int io, cudaStream_t st) {
  if (rows < 1 || V < 1) return SL_ERR_BAD_SHAPE;
  const int w = io == SL_F32 ? 4 : 8;
  SL_DISPATCH_DTYPE(io, T, SL_VEC_DISPATCH(V % w == 0 && aligned(logits, 16) && aligned(d, 16), {
    ce_bwd_kernel<T, VEC><<<(unsigned)rows, row_threads(V / w), 0, st>>>(reinterpret_cast<const T*>(logits), target, lse, g, scale,
                                                                         reinterpret_cast<T*>(d), V);
  }));
  note_launches(1);
  return launch_status();
}
int embedding_bwd(const int* sorted, const int64_t* order, const void* d_out, void* dE, int n, int V, int C, int io,
                  cudaStream_t st) {
  if (V < 1 || C < 1) return SL_ERR_BAD_SHAPE;
  const int w = io == SL_F32 ? 4 : 8;
  SL_DISPATCH_DTYPE(io, T, SL_VEC_DISPATCH(C % w == 0 && aligned(d_out, 16) && aligned(dE, 16), {
    const int pieces = VEC ? C / w : C;
    embedding_bwd_kernel<T, VEC><<<(unsigned)V, pieces >= 256 ? 256 : pieces >= 128 ? 128 : 64, 0, st>>>(
        sorted, order, reinterpret_cast<const T*>(d_out), reinterpret_cast<T*>(dE), n, C);
  }));
  note_launches(1);
  return launch_status();
}

unsigned mt_chunks(int64_t len) { return (unsigned)((len + MT_CHUNK - 1) / MT_CHUNK); }
int multi_sumsq(const MtList1& list, unsigned chunks, float* partial, int io, cudaStream_t st) {
  SL_DISPATCH_DTYPE(io, T, { sumsq_kernel<T><<<chunks, 256, 0, st>>>(list, partial); });
  note_launches(1);
  return launch_status();
}
int norm_finish(const float* partial, int n, float clip, float* out, cudaStream_t st) {
  norm_finish_kernel<<<1, 1024, 0, st>>>(partial, n, clip, out);
  note_launches(1);
  return launch_status();
}
int multi_adamw(const MtList4& list, unsigned chunks, const AdamWArgs& a, int io, cudaStream_t st) {
  SL_DISPATCH_DTYPE(io, T, { adamw_kernel<T><<<chunks, 256, 0, st>>>(list, a); });
  note_launches(1);
  return launch_status();
}

}  // namespace sl
