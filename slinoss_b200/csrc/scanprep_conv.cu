// Scan preparation fused with the causal depthwise conv1d + SiLU of the value stream.
//
// Forward (one C-ABI call, three coalesced elementwise kernels on one stream):
//   value kernel  out[b,t,c] = SiLU(bias_c + sum_j W[c,j] x[b,t-(d_conv-1)+j,c]) written
//                 straight into the (batch,heads,T,P) layout of U
//                 (reference: slinoss/ops/mixer/convolution.py:68-101 followed by the
//                 transpose of slinoss/layers/scanprep.py:307-321)
//   bc kernel     amplitude = softplus, phase = pi*tanh, pair = amp*(cos,sin)/rms_n(amp)
//                 (slinoss/ops/scanprep/parameterization.py:45-107)
//   coeff kernel  dt/alpha/theta maps, rho = r e^{i theta}, exact first-order-hold taps
//                 (slinoss/layers/scanprep.py:237-283, slinoss/ops/scanprep/reference.py:25-56)
// The tap formulas cancel catastrophically in float32 for small |z| (the
// numerator of kappa2 loses ~1/|z|^2 ulps), so the coefficient kernels evaluate them
// in float64; the count is one complex per (batch, head, token), which is negligible.
//
// Backward mirrors the three kernels; parameter-bias and conv weight/bias
// gradients are reduced per CTA and accumulated with float atomics.
#include <type_traits>

#include <mutex>

#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

#include "scanprep_math.cuh"

constexpr int CONV_TT = 32;  // tokens per CTA in the value kernels

template <typename T> __device__ __forceinline__ void load4(const T* p, float (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
  } else {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = unpack_pair<T>(r.x), b = unpack_pair<T>(r.y);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}
template <typename T> __device__ __forceinline__ void store4(T* p, const float (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_pair<T>(v[0], v[1]), pack_pair<T>(v[2], v[3]));
  }
}

struct ValueParams {
  const void *x, *w, *bias, *state_in;
  void *state_out, *U;
  int64_t xs;                   // row stride of x (elements)
  int64_t usb, ush, ust;        // strides of U
  int batch, T, C, P, W;
};

template <typename T>
__device__ __forceinline__ float load_x(const ValueParams& p, const T* x, const T* st, int b,
                                        int t, int c) {
  // input at time t (t may be negative: carried conv state or zero)
  if (t >= 0) return to_f32(x[((size_t)b * p.T + t) * p.xs + c]);
  const int j = p.W - 1 + t;
  if (st && j >= 0) return to_f32(st[((size_t)b * p.C + c) * (p.W - 1) + j]);
  return 0.f;
}

template <typename T>
__global__ void __launch_bounds__(256) value_fwd_kernel(ValueParams p) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int t0 = blockIdx.y * CONV_TT, b = blockIdx.z;
  if (c >= p.C) return;
  const T* x = reinterpret_cast<const T*>(p.x);
  const T* st = reinterpret_cast<const T*>(p.state_in);
  T* U = reinterpret_cast<T*>(p.U);
  const int h = c / p.P, pp = c - h * p.P;
  const int t1 = min(t0 + CONV_TT, p.T);
  if (!p.w) {
    for (int t = t0; t < t1; ++t)
      U[(size_t)b * p.usb + (size_t)h * p.ush + (size_t)t * p.ust + pp] =
          x[((size_t)b * p.T + t) * p.xs + c];
    return;
  }
  const T* w = reinterpret_cast<const T*>(p.w);
  float wj[4] = {0.f, 0.f, 0.f, 0.f}, win[4] = {0.f, 0.f, 0.f, 0.f};
  // right-align the taps in a width-4 window: wj[4-W+j] = W[c][j]
  for (int j = 0; j < p.W; ++j) wj[4 - p.W + j] = to_f32(w[(size_t)c * p.W + j]);
  const float bias = p.bias ? to_f32(reinterpret_cast<const T*>(p.bias)[c]) : 0.f;
  // win[k] holds x at time t-3+k
  for (int k = 1; k < 4; ++k) win[k] = (4 - k <= p.W - 1) ? load_x(p, x, st, b, t0 - 4 + k, c) : 0.f;
  for (int t = t0; t < t1; ++t) {
    win[0] = win[1]; win[1] = win[2]; win[2] = win[3];
    win[3] = to_f32(x[((size_t)b * p.T + t) * p.xs + c]);
    const float a = bias + wj[0] * win[0] + wj[1] * win[1] + wj[2] * win[2] + wj[3] * win[3];
    U[(size_t)b * p.usb + (size_t)h * p.ush + (size_t)t * p.ust + pp] = from_f32<T>(silu_f(a));
  }
  if (p.state_out && t1 == p.T) {
    T* so = reinterpret_cast<T*>(p.state_out);
    for (int j = 0; j < p.W - 1; ++j)
      so[((size_t)b * p.C + c) * (p.W - 1) + j] =
          from_f32<T>(load_x(p, x, st, b, p.T - (p.W - 1) + j, c));
  }
}

struct ValueBwdParams {
  ValueParams f;
  const void* dU;
  void *dx, *dstate;
  int64_t dxs;                  // row stride of dx
  const void* dY;               // optional, laid out like dU: the gradient of U is dU + skip[head] * dY
  const float* skip;
  float *dw, *dbias;
};

__device__ __forceinline__ float dsilu_f(float a) {
  const float s = sigmoid_f(a);
  return s * (1.f + a * (1.f - s));
}

// One thread per channel walks CONV_TT tokens; da at tokens t..t+W-1 is needed
// for dx[t], so da is recomputed over a (W-1)-token look-ahead halo.
template <typename T>
__global__ void __launch_bounds__(256) value_bwd_kernel(ValueBwdParams q) {
  const ValueParams& p = q.f;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int t0 = blockIdx.y * CONV_TT, b = blockIdx.z;
  if (c >= p.C) return;
  const T* x = reinterpret_cast<const T*>(p.x);
  const T* st = reinterpret_cast<const T*>(p.state_in);
  const T* dU = reinterpret_cast<const T*>(q.dU);
  T* dx = reinterpret_cast<T*>(q.dx);
  const int h = c / p.P, pp = c - h * p.P;
  const int t1 = min(t0 + CONV_TT, p.T);
  auto dy_at = [&](int t) -> float {
    const size_t i = (size_t)b * p.usb + (size_t)h * p.ush + (size_t)t * p.ust + pp;
    return to_f32(dU[i]) + (q.dY ? q.skip[h] * to_f32(reinterpret_cast<const T*>(q.dY)[i]) : 0.f);
  };
  if (!p.w) {
    for (int t = t0; t < t1; ++t) dx[((size_t)b * p.T + t) * q.dxs + c] = from_f32<T>(dy_at(t));
    return;
  }
  const T* w = reinterpret_cast<const T*>(p.w);
  const int W = p.W;
  float wj[4] = {0.f, 0.f, 0.f, 0.f};
  for (int j = 0; j < W; ++j) wj[4 - W + j] = to_f32(w[(size_t)c * W + j]);
  const float bias = p.bias ? to_f32(reinterpret_cast<const T*>(p.bias)[c]) : 0.f;
  float win[4] = {0.f, 0.f, 0.f, 0.f};   // x at times s-3..s for the da being formed
  float da[4] = {0.f, 0.f, 0.f, 0.f};    // da at times s-3..s
  float dwacc[4] = {0.f, 0.f, 0.f, 0.f}, dbacc = 0.f;
  // The first tile also owns the gradient of the carried conv state (times < 0).
  const int s_begin = (t0 == 0) ? 0 : t0;
  for (int k = 1; k < 4; ++k) win[k] = (4 - k <= W - 1) ? load_x(p, x, st, b, s_begin - 4 + k, c) : 0.f;
  // s runs over the tokens whose da is formed; dx[s-3] becomes complete at step s
  // when W == 4 (in general dx[t] needs da[t .. t+W-1]).
  const int s_end = min(t1 + 3, p.T + 3);
  for (int s = s_begin; s < s_end; ++s) {
    win[0] = win[1]; win[1] = win[2]; win[2] = win[3];
    da[0] = da[1]; da[1] = da[2]; da[2] = da[3];
    float d = 0.f;
    if (s < p.T) {
      win[3] = to_f32(x[((size_t)b * p.T + s) * p.xs + c]);
      const float a = bias + wj[0] * win[0] + wj[1] * win[1] + wj[2] * win[2] + wj[3] * win[3];
      d = dy_at(s) * dsilu_f(a);
      if (s >= t0 && s < t1) {  // each token's weight/bias contribution is counted once
        dwacc[0] += d * win[0]; dwacc[1] += d * win[1];
        dwacc[2] += d * win[2]; dwacc[3] += d * win[3];
        dbacc += d;
      }
    } else {
      win[3] = 0.f;
    }
    da[3] = d;
    // dx[t] = sum_k wj[k] * da[t + 3 - k], complete for t = s - 3
    const int t = s - 3;
    const float g = wj[3] * da[0] + wj[2] * da[1] + wj[1] * da[2] + wj[0] * da[3];
    if (t >= t0 && t < t1) dx[((size_t)b * p.T + t) * q.dxs + c] = from_f32<T>(g);
    else if (t < 0 && t0 == 0 && q.dstate && t >= -(W - 1))
      reinterpret_cast<T*>(q.dstate)[((size_t)b * p.C + c) * (W - 1) + (W - 1 + t)] = from_f32<T>(g);
  }
  for (int j = 0; j < W; ++j) atomicAdd(q.dw + (size_t)c * W + j, dwacc[4 - W + j]);
  if (q.dbias) atomicAdd(q.dbias + c, dbacc);
}

// ---- vector path of the value kernels ----------------------------------------------------------------
// A thread owns 4 consecutive channels (one 8- or 16-byte access per token) and walks CONV_TT
// tokens; a warp covers 128 consecutive channels, a CTA of 256 threads 8 token sub-tiles of the
// same 128 channels, so that the conv weight / bias gradients of the 8 sub-tiles are combined in
// shared memory and added to the float32 accumulators once per CTA.
// Needs P % 4 == 0 (a piece stays inside one head), strides that are multiples of 4 and aligned
// pointers; anything else takes the one-channel-per-thread kernels above.
constexpr int CONV_V = 4;
constexpr int CONV_SUB = 8;   // token sub-tiles per CTA
constexpr int CONV_SB = 4;    // tokens of a batch

template <typename T>
__device__ __forceinline__ void load_xv(const ValueParams& p, const T* x, const T* st, int b, int t, int c,
                                        float (&v)[CONV_V]) {
  if (t >= 0) { load4<T>(x + ((size_t)b * p.T + t) * p.xs + c, v); return; }
  const int j = p.W - 1 + t;
#pragma unroll
  for (int k = 0; k < CONV_V; ++k)
    v[k] = (st && j >= 0) ? to_f32(st[((size_t)b * p.C + c + k) * (p.W - 1) + j]) : 0.f;
}

// 4 channels as two packed pairs, and the memory piece they come in
template <typename T> using Raw4 = typename std::conditional<sizeof(T) == 4, uint4, uint2>::type;
template <typename T> __device__ __forceinline__ void unpack4(const Raw4<T>& r, f2 (&v)[2]) {
  if constexpr (sizeof(T) == 4) {
    v[0] = mk2(__uint_as_float(r.x), __uint_as_float(r.y));
    v[1] = mk2(__uint_as_float(r.z), __uint_as_float(r.w));
  } else {
    const float2 a = unpack_pair<T>(r.x), b = unpack_pair<T>(r.y);
    v[0] = mk2(a.x, a.y); v[1] = mk2(b.x, b.y);
  }
}
template <typename T> __device__ __forceinline__ void store4(T* p, const f2 (&v)[2]) {
  const float2 a = un2(v[0]), b = un2(v[1]);
  const float q[4] = {a.x, a.y, b.x, b.y};
  store4<T>(p, q);
}

// The taps, right-aligned in a window of 4, the bias, and the 3 inputs before token t0 (those that no tap reads as zeros) of
// the channels c .. c + 3.
template <typename T>
__device__ __forceinline__ void conv_setup(const ValueParams& p, int b, int t0, int c, f2 (&w2)[4][2], f2 (&bias2)[2],
                                           f2 (&win)[3][2]) {
  const T *w = reinterpret_cast<const T*>(p.w), *x = reinterpret_cast<const T*>(p.x), *st = reinterpret_cast<const T*>(p.state_in);
  float wj[4][CONV_V], bias[CONV_V] = {0.f, 0.f, 0.f, 0.f}, h[CONV_V];
  if (p.W == 4 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
    // the taps of the 4 channels are 16 contiguous values; bias is one 4-wide piece
#pragma unroll
    for (int k = 0; k < CONV_V; ++k) {
      float q[4];
      load4<T>(w + (size_t)(c + k) * 4, q);
#pragma unroll
      for (int j = 0; j < 4; ++j) wj[j][k] = q[j];
    }
    if (p.bias) load4<T>(reinterpret_cast<const T*>(p.bias) + c, bias);
  } else {
#pragma unroll
    for (int k = 0; k < CONV_V; ++k) {
#pragma unroll
      for (int j = 0; j < 4; ++j) wj[j][k] = (j >= 4 - p.W) ? to_f32(w[(size_t)(c + k) * p.W + (j - (4 - p.W))]) : 0.f;
      if (p.bias) bias[k] = to_f32(reinterpret_cast<const T*>(p.bias)[c + k]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w2[j][i] = mk2(wj[j][2 * i], wj[j][2 * i + 1]);
    bias2[i] = mk2(bias[2 * i], bias[2 * i + 1]);
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    win[r][0] = win[r][1] = 0;
    if (3 - r > p.W - 1) continue;
    load_xv<T>(p, x, st, b, t0 - 3 + r, c, h);
    win[r][0] = mk2(h[0], h[1]); win[r][1] = mk2(h[2], h[3]);
  }
}

// Forward.  Each batch of 4 tokens is requested one batch ahead of its use: the loads of a batch alone (3 KB per warp and
// latency, as the walk alternated between waiting and computing) left two thirds of the bandwidth idle.
template <typename T>
__global__ void __launch_bounds__(256, 3) value_fwd_vec_kernel(ValueParams p, int tile) {
  const int c = (blockIdx.x * 32 + (threadIdx.x & 31)) * CONV_V;
  const int t0 = (blockIdx.y * CONV_SUB + (threadIdx.x >> 5)) * tile, b = blockIdx.z;
  if (c >= p.C || t0 >= p.T) return;
  const int h = c / p.P, pp = c - h * p.P, t1 = min(t0 + tile, p.T);
  T* Ub = reinterpret_cast<T*>(p.U) + (size_t)b * p.usb + (size_t)h * p.ush + pp;
  const T* xb = reinterpret_cast<const T*>(p.x) + (size_t)b * p.T * p.xs + c;
  Raw4<T> nx[CONV_SB];
  auto fetch = [&](int s) {
#pragma unroll
    for (int i = 0; i < CONV_SB; ++i)
      if (s + i < p.T) nx[i] = *reinterpret_cast<const Raw4<T>*>(xb + (size_t)(s + i) * p.xs);
  };
  fetch(t0);
  if (!p.w) {
    for (int s = t0; s < t1; s += CONV_SB) {
      Raw4<T> cx[CONV_SB];
#pragma unroll
      for (int i = 0; i < CONV_SB; ++i) cx[i] = nx[i];
      if (s + CONV_SB < t1) fetch(s + CONV_SB);
#pragma unroll
      for (int i = 0; i < CONV_SB; ++i)
        if (s + i < t1) *reinterpret_cast<Raw4<T>*>(Ub + (size_t)(s + i) * p.ust) = cx[i];
    }
    return;
  }
  f2 w[4][2], bias[2], win[3][2];
  conv_setup<T>(p, b, t0, c, w, bias, win);
#pragma unroll 1
  for (int s = t0; s < t1; s += CONV_SB) {
    Raw4<T> cx[CONV_SB];
#pragma unroll
    for (int i = 0; i < CONV_SB; ++i) cx[i] = nx[i];
    if (s + CONV_SB < t1) fetch(s + CONV_SB);
#pragma unroll
    for (int i = 0; i < CONV_SB; ++i) {
      f2 x[2], o[2];
      unpack4<T>(cx[i], x);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const f2 a = fma2(w[3][k], x[k], fma2(w[2][k], win[2][k], fma2(w[1][k], win[1][k], fma2(w[0][k], win[0][k], bias[k]))));
        o[k] = mul2(a, sigmoid2(a));
        win[0][k] = win[1][k]; win[1][k] = win[2][k]; win[2][k] = x[k];
      }
      if (s + i < t1) store4<T>(Ub + (size_t)(s + i) * p.ust, o);
    }
  }
  if (p.state_out && t1 == p.T) {
    T* so = reinterpret_cast<T*>(p.state_out);
    for (int j = 0; j < p.W - 1; ++j) {
      float v[CONV_V];
      load_xv<T>(p, reinterpret_cast<const T*>(p.x), reinterpret_cast<const T*>(p.state_in), b, p.T - (p.W - 1) + j, c, v);
#pragma unroll
      for (int k = 0; k < CONV_V; ++k) so[((size_t)b * p.C + c + k) * (p.W - 1) + j] = from_f32<T>(v[k]);
    }
  }
}

// Backward.  Bound by the instructions per channel and token (about 20 in packed pairs; 53 before) and by the latency of a
// batch, which is requested one batch ahead.  A tile of n tokens walks n + 3 steps: the last three only complete dx.
// (8, 2048) tokens of 2048 channels: 103 -> 71 us; (1, 1021), where the ragged last tile used to walk token by token: 42 -> 17
// (forward 23 -> 10).
template <typename T, bool SKIP>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 2 : 1) value_bwd_vec_kernel(ValueBwdParams q, int tile) {
  const ValueParams& p = q.f;
  constexpr int ROW = 32 * CONV_V + 8;              // 8 floats of padding: the sums below read 4 rows side by side
  __shared__ float s_acc[CONV_SUB][5][ROW];         // dw (4 taps) and dbias partials per sub-tile
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * CONV_V;
  const int t0 = (blockIdx.y * CONV_SUB + sub) * tile, b = blockIdx.z, t1 = min(t0 + tile, p.T);
  f2 dw[4][2], db[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    db[k] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) dw[j][k] = 0;
  }
  if (c < p.C && t0 < p.T) {
    const int h = c / p.P, pp = c - h * p.P;
    const size_t ub = (size_t)b * p.usb + (size_t)h * p.ush + pp;
    const T* xb = reinterpret_cast<const T*>(p.x) + (size_t)b * p.T * p.xs + c;
    const T* dUb = reinterpret_cast<const T*>(q.dU) + ub;
    const T* dYb = SKIP ? reinterpret_cast<const T*>(q.dY) + ub : nullptr;
    T* dxb = reinterpret_cast<T*>(q.dx) + (size_t)b * p.T * q.dxs + c;
    const f2 skip = SKIP ? dup2(q.skip[h]) : 0;
    Raw4<T> nx[CONV_SB], ng[CONV_SB], ny[SKIP ? CONV_SB : 1];
    auto fetch = [&](int s) {      // tokens past the end count as zeros
#pragma unroll
      for (int i = 0; i < CONV_SB; ++i) {
        nx[i] = ng[i] = Raw4<T>{};
        if constexpr (SKIP) ny[i] = Raw4<T>{};
        if (s + i >= p.T) continue;
        nx[i] = *reinterpret_cast<const Raw4<T>*>(xb + (size_t)(s + i) * p.xs);
        ng[i] = *reinterpret_cast<const Raw4<T>*>(dUb + (size_t)(s + i) * p.ust);
        if constexpr (SKIP) ny[i] = *reinterpret_cast<const Raw4<T>*>(dYb + (size_t)(s + i) * p.ust);
      }
    };
    auto gradient = [&](const Raw4<T>& g, const Raw4<T>& y, f2 (&v)[2]) {
      unpack4<T>(g, v);
      if constexpr (SKIP) {
        f2 yv[2];
        unpack4<T>(y, yv);
        v[0] = fma2(skip, yv[0], v[0]); v[1] = fma2(skip, yv[1], v[1]);
      }
    };
    fetch(t0);
    if (!p.w) {
      for (int s = t0; s < t1; s += CONV_SB) {
        f2 v[CONV_SB][2];
#pragma unroll
        for (int i = 0; i < CONV_SB; ++i) gradient(ng[i], ny[SKIP ? i : 0], v[i]);
        if (s + CONV_SB < t1) fetch(s + CONV_SB);
#pragma unroll
        for (int i = 0; i < CONV_SB; ++i)
          if (s + i < t1) store4<T>(dxb + (size_t)(s + i) * q.dxs, v[i]);
      }
    } else {
      const int W = p.W;
      f2 w[4][2], bias[2], win[3][2], da[3][2];
      conv_setup<T>(p, b, t0, c, w, bias, win);
#pragma unroll
      for (int k = 0; k < 2; ++k) da[0][k] = da[1][k] = da[2][k] = 0;
      // da of token s; dx[s-3] is complete at step s.  ``mine``: the token's weight / bias contribution is counted here
      auto step = [&](int s, auto mine, const f2 (&x)[2], const f2 (&gy)[2]) {
        f2 g[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const f2 a = fma2(w[3][k], x[k], fma2(w[2][k], win[2][k], fma2(w[1][k], win[1][k], fma2(w[0][k], win[0][k], bias[k]))));
          const f2 sg = sigmoid2(a), one = dup2(1.f);
          const f2 d = mul2(gy[k], mul2(sg, fma2(a, fma2(sg, dup2(-1.f), one), one)));
          if constexpr (decltype(mine)::value) {
            dw[0][k] = fma2(d, win[0][k], dw[0][k]); dw[1][k] = fma2(d, win[1][k], dw[1][k]);
            dw[2][k] = fma2(d, win[2][k], dw[2][k]); dw[3][k] = fma2(d, x[k], dw[3][k]);
            db[k] = add2(db[k], d);
          }
          g[k] = fma2(w[0][k], d, fma2(w[1][k], da[2][k], fma2(w[2][k], da[1][k], mul2(w[3][k], da[0][k]))));
          win[0][k] = win[1][k]; win[1][k] = win[2][k]; win[2][k] = x[k];
          da[0][k] = da[1][k]; da[1][k] = da[2][k]; da[2][k] = d;
        }
        const int t = s - 3;
        if (t >= t0) {
          if (t < t1) store4<T>(dxb + (size_t)t * q.dxs, g);
        } else if (q.dstate && t < 0 && t >= -(W - 1)) {   // the first tile also owns the gradient of the carried conv state
          const float2 lo = un2(g[0]), hi = un2(g[1]);
          const float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
          for (int k = 0; k < CONV_V; ++k)
            reinterpret_cast<T*>(q.dstate)[((size_t)b * p.C + c + k) * (W - 1) + (W - 1 + t)] = from_f32<T>(v[k]);
        }
      };
      auto batch = [&](int s, auto mine, bool more) {
        constexpr int n = decltype(mine)::value ? CONV_SB : 3;
        Raw4<T> cx[n], cg[n], cy[SKIP ? n : 1];
#pragma unroll
        for (int i = 0; i < n; ++i) { cx[i] = nx[i]; cg[i] = ng[i]; if constexpr (SKIP) cy[i] = ny[i]; }
        if (more) fetch(s + CONV_SB);
#pragma unroll
        for (int i = 0; i < n; ++i) {
          f2 x[2], gy[2];
          unpack4<T>(cx[i], x);
          gradient(cg[i], cy[SKIP ? i : 0], gy);
          step(s + i, mine, x, gy);
        }
      };
      int s = t0;
#pragma unroll 1
      for (; s < t1; s += CONV_SB) batch(s, std::true_type{}, true);
      batch(s, std::false_type{}, false);
    }
  }
  if (!p.w) return;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int j = 0; j < 5; ++j) *reinterpret_cast<f2*>(&s_acc[sub][j][lane * CONV_V + 2 * k]) = j < 4 ? dw[j & 3][k] : db[k];
  }
  __syncthreads();
  // 5 x 128 sums of CONV_SUB partials; one atomic per (channel, tap) per CTA, the taps of a channel side by side
  for (int i = threadIdx.x; i < 5 * 32 * CONV_V; i += blockDim.x) {
    const int j = i < 4 * 32 * CONV_V ? i & 3 : 4, cc = j < 4 ? i >> 2 : i - 4 * 32 * CONV_V;
    const int ch = blockIdx.x * 32 * CONV_V + cc;
    if (ch >= p.C) continue;
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < CONV_SUB; ++r) v += s_acc[r][j][cc];
    if (j < 4) { if (j >= 4 - p.W) atomicAdd(q.dw + (size_t)ch * p.W + (j - (4 - p.W)), v); }
    else if (q.dbias) atomicAdd(q.dbias + ch, v);
  }
}

// Tokens per warp: 32 (the walk restarts at a tile with 3 tokens of its neighbour), shorter while that leaves fewer than two
// CTAs per SM - a warp walks its tile at one load latency per 4 tokens, 18 us for 32 of them.
inline int conv_tile(int T, int C, int batch) {
  int tile = 32;
  const long long columns = (long long)batch * ((C + 32 * CONV_V - 1) / (32 * CONV_V));
  while (tile > 8 && columns * ((T + CONV_SUB * tile - 1) / (CONV_SUB * tile)) < 2 * 148) tile /= 2;
  return tile;
}

inline bool value_vec_ok(const ValueParams& p, const void* a, const void* b) {
  constexpr int align = 16, V = CONV_V;
  return p.P % V == 0 && p.C % V == 0 && p.xs % V == 0 && p.usb % V == 0 &&
         p.ush % V == 0 && p.ust % V == 0 && aligned(p.x, align) && aligned(p.U, align) &&
         (a == nullptr || aligned(a, align)) && (b == nullptr || aligned(b, align));
}

// ---- B / C parameterisation ------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(256) bc_fwd_kernel(const T* __restrict__ bc, T* __restrict__ Bo,
                                                     T* __restrict__ Co, int64_t bcs, int batch, int Tn,
                                                     int G, int N, float eps) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= (long long)batch * Tn * G) return;
  const int g = (int)(row % G);
  const long long bt = row / G;
  const int t = (int)(bt % Tn), b = (int)(bt / Tn);
  const T* src = bc + (size_t)bt * bcs + (size_t)g * 4 * N;
  T* outs[2] = {Bo + (((size_t)b * G + g) * Tn + t) * 2 * N, Co + (((size_t)b * G + g) * Tn + t) * 2 * N};
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const T* amp_row = src + (size_t)(2 * which) * N;
    const T* ph_row = amp_row + N;
    float ss = 0.f;
    for (int n = lane; n < N; n += 32) {
      const float a = softplus_f(to_f32(amp_row[n]));
      ss += a * a;
    }
    ss = warp_sum(ss);
    const float inv = rsqrtf(fmaxf(ss / (float)N, eps));
    for (int n = lane; n < N; n += 32) {
      const float a = softplus_f(to_f32(amp_row[n])) * inv;
      const float ph = 3.14159265358979323846f * tanhf(to_f32(ph_row[n]));
      float sn, cs;
      sincosf(ph, &sn, &cs);
      outs[which][2 * n] = from_f32<T>(a * cs);
      outs[which][2 * n + 1] = from_f32<T>(a * sn);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) bc_bwd_kernel(const T* __restrict__ bc,
                                                     const T* __restrict__ dBo,
                                                     const T* __restrict__ dCo,
                                                     T* __restrict__ dbc, int64_t bcs, int64_t dbcs, int batch,
                                                     int Tn, int G, int N, float eps) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= (long long)batch * Tn * G) return;
  const int g = (int)(row % G);
  const long long bt = row / G;
  const int t = (int)(bt % Tn), b = (int)(bt / Tn);
  const T* src = bc + (size_t)bt * bcs + (size_t)g * 4 * N;
  T* dst = dbc + (size_t)bt * dbcs + (size_t)g * 4 * N;
  const T* gs[2] = {dBo + (((size_t)b * G + g) * Tn + t) * 2 * N, dCo + (((size_t)b * G + g) * Tn + t) * 2 * N};
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const T* amp_row = src + (size_t)(2 * which) * N;
    const T* ph_row = amp_row + N;
    float ss = 0.f, gsum = 0.f;
    for (int n = lane; n < N; n += 32) {
      const float a = softplus_f(to_f32(amp_row[n]));
      const float ph = 3.14159265358979323846f * tanhf(to_f32(ph_row[n]));
      float sn, cs;
      sincosf(ph, &sn, &cs);
      ss += a * a;
      gsum += a * (cs * to_f32(gs[which][2 * n]) + sn * to_f32(gs[which][2 * n + 1]));
    }
    ss = warp_sum(ss); gsum = warp_sum(gsum);
    const float ms = ss / (float)N;
    const float inv = rsqrtf(fmaxf(ms, eps));
    const float g_ms = ms > eps ? -0.5f * inv * inv * inv * gsum : 0.f;
    for (int n = lane; n < N; n += 32) {
      const float xa = to_f32(amp_row[n]);
      const float a = softplus_f(xa);
      const float th = tanhf(to_f32(ph_row[n]));
      const float ph = 3.14159265358979323846f * th;
      float sn, cs;
      sincosf(ph, &sn, &cs);
      const float gre = to_f32(gs[which][2 * n]), gim = to_f32(gs[which][2 * n + 1]);
      const float g_amp = inv * (cs * gre + sn * gim) + g_ms * 2.f * a / (float)N;
      const float g_ph = a * inv * (cs * gim - sn * gre);
      dst[(size_t)(2 * which) * N + n] = from_f32<T>(g_amp * sigmoid_f(xa));
      dst[(size_t)(2 * which + 1) * N + n] = from_f32<T>(g_ph * 3.14159265358979323846f * (1.f - th * th));
    }
  }
}

// ---- vector path of the B / C kernels (N % 4 == 0, N <= 128) ---------------------------------------
// One warp per (batch, token, group) record of 4 rows x N: lanes 0-15 produce B, lanes 16-31 C (N <= 64), or
// two neighbouring warps, one for B and one for C (WIDE, N <= 128: the one-element-per-lane kernels above took
// 53 us for 1021 tokens x 32 groups x 128);
// a lane owns 4 consecutive n: two 8-byte loads (amplitude and phase logits), one 16-byte store of
// 4 complex values.  The mean over n is a shuffle reduction inside the lanes of B or C.  With 16-bit
// io the transcendental functions are the fast intrinsics (their error is far below the output's
// rounding); float32 io keeps the precise ones.
template <bool FAST> __device__ __forceinline__ float tanh_v(float x) {
  if (FAST) {   // PTX tanh.approx, relative error 2^-11: below the rounding of 16-bit outputs
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  }
  return tanhf(x);
}
template <bool FAST> __device__ __forceinline__ void sincos_v(float x, float* s, float* c) {
  if (FAST) __sincosf(x, s, c);   // |x| <= pi here
  else sincosf(x, s, c);
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float (&v)[8]) {
  if constexpr (sizeof(T) == 2) {
    store16<T>(p, v);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float4*>(p + 4 * h) = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
  }
}
template <bool WIDE> __device__ __forceinline__ float part_sum(float v) {   // over the 16 (WIDE: 32) lanes of B or C
#pragma unroll
  for (int o = WIDE ? 16 : 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int BC_GCH = 8;   // groups one warp walks: grid = (tokens / 8, groups / BC_GCH, batch)

// Pairs of the maps above.  The 16-bit forms are softplus x = max(x, 0) + ln(1 + e^-|x|) with e^x = 2^(x log2 e) and
// ln x = ln 2 log2 x on the PTX instructions ex2.approx and lg2.approx.
template <bool FAST> __device__ __forceinline__ f2 softplus2(f2 x) {
  const float2 v = un2(x);
  if constexpr (!FAST) return mk2(softplus_f(v.x), softplus_f(v.y));
  const f2 e = mk2(ex2f(-1.4426950408889634f * fabsf(v.x)), ex2f(-1.4426950408889634f * fabsf(v.y)));
  const float2 d = un2(add2(e, dup2(1.f)));
  return fma2(mk2(lg2f(d.x), lg2f(d.y)), dup2(0.6931471805599453f), mk2(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f)));
}
template <bool FAST> __device__ __forceinline__ f2 tanh2(f2 x) {
  const float2 v = un2(x);
  return mk2(tanh_v<FAST>(v.x), tanh_v<FAST>(v.y));
}
template <bool FAST> __device__ __forceinline__ f2 sigmoid_pair(f2 x) {
  if constexpr (FAST) return fma2(tanh2<true>(mul2(x, dup2(0.5f))), dup2(0.5f), dup2(0.5f));
  const float2 v = un2(x);
  return mk2(sigmoid_f(v.x), sigmoid_f(v.y));
}
template <bool FAST> __device__ __forceinline__ void sincos2(f2 x, f2* s, f2* c) {
  const float2 v = un2(x);
  float2 a, b;
  sincos_v<FAST>(v.x, &a.x, &b.x); sincos_v<FAST>(v.y, &a.y, &b.y);
  *s = mk2(a.x, a.y); *c = mk2(b.x, b.y);
}
// 4 complex values (re, im interleaved) as two pairs of real and two of imaginary parts, and their memory pieces
template <typename T> struct Raw8 { Raw4<T> lo, hi; };
template <typename T> __device__ __forceinline__ Raw8<T> load_raw8(const T* p) {
  if constexpr (sizeof(T) == 2) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    return {make_uint2(q.x, q.y), make_uint2(q.z, q.w)};
  } else {
    return {*reinterpret_cast<const uint4*>(p), *reinterpret_cast<const uint4*>(p + 4)};
  }
}
template <typename T> __device__ __forceinline__ void split8(const Raw8<T>& r, f2 (&re)[2], f2 (&im)[2]) {
  f2 q[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    unpack4<T>(h ? r.hi : r.lo, q);
    const float2 a = un2(q[0]), b = un2(q[1]);
    re[h] = mk2(a.x, b.x); im[h] = mk2(a.y, b.y);
  }
}

// One warp per (batch, token, run of up to BC_GCH groups); the grid carries batch and the run, so no
// index is divided at run time.  The next record's logits are requested before the current one is
// evaluated.  Bound by the special-function unit (five operations per complex pair, 74 us of it in 16384 tokens x 32 groups x
// N = 64 against 83 of DRAM) once the rest is in
// packed pairs: 115 -> 96 us, the backward 197 -> 154 (DRAM 125).
template <typename T, bool WIDE>
__global__ void __launch_bounds__(256) bc_fwd_vec_kernel(const T* __restrict__ bc, T* __restrict__ Bo,
                                                         T* __restrict__ Co, int64_t bcs, int Tn, int G, int N, float eps) {
  constexpr bool FAST = sizeof(T) == 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int which = WIDE ? warp & 1 : lane >> 4, n0 = 4 * (WIDE ? lane : lane & 15);
  const int t = WIDE ? blockIdx.x * 4 + (warp >> 1) : blockIdx.x * 8 + warp, b = blockIdx.z;
  const int g0 = blockIdx.y * BC_GCH, g1 = min(G, g0 + BC_GCH);
  if (t >= Tn) return;
  const bool act = n0 < N;
  const T* src = bc + ((size_t)b * Tn + t) * bcs + (size_t)(4 * g0 + 2 * which) * N + n0;
  T* dst = (which ? Co : Bo) + (((size_t)b * G + g0) * Tn + t) * 2 * N + 2 * n0;
  const size_t dstep = (size_t)Tn * 2 * N;
  const float inv_n = 1.f / (float)N;
  Raw4<T> na{}, np{};
  auto fetch = [&] {
    if (!act) return;
    na = *reinterpret_cast<const Raw4<T>*>(src);
    np = *reinterpret_cast<const Raw4<T>*>(src + N);
  };
  fetch();
#pragma unroll 2
  for (int g = g0; g < g1; ++g) {
    f2 amp[2], ph[2];
    unpack4<T>(na, amp); unpack4<T>(np, ph);
    src += 4 * N;
    if (g + 1 < g1) fetch();
    amp[0] = softplus2<FAST>(amp[0]); amp[1] = softplus2<FAST>(amp[1]);
    const float2 sq = un2(fma2(amp[0], amp[0], mul2(amp[1], amp[1])));
    const float ss = part_sum<WIDE>(act ? sq.x + sq.y : 0.f);
    if (act) {
      const f2 inv = dup2(rsqrtf(fmaxf(ss * inv_n, eps)));
      float o[8];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        f2 sn, cs;
        sincos2<FAST>(mul2(tanh2<FAST>(ph[i]), dup2(3.14159265358979323846f)), &sn, &cs);
        const f2 a = mul2(amp[i], inv);
        const float2 re = un2(mul2(a, cs)), im = un2(mul2(a, sn));
        o[4 * i] = re.x; o[4 * i + 1] = im.x; o[4 * i + 2] = re.y; o[4 * i + 3] = im.y;
      }
      store8<T>(dst, o);
    }
    dst += dstep;
  }
}

template <typename T, bool WIDE>
__global__ void __launch_bounds__(256) bc_bwd_vec_kernel(const T* __restrict__ bc,
                                                         const T* __restrict__ dBo,
                                                         const T* __restrict__ dCo,
                                                         T* __restrict__ dbc, int64_t bcs, int64_t dbcs, int Tn, int G,
                                                         int N, float eps) {
  constexpr bool FAST = sizeof(T) == 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int which = WIDE ? warp & 1 : lane >> 4, n0 = 4 * (WIDE ? lane : lane & 15);
  const int t = WIDE ? blockIdx.x * 4 + (warp >> 1) : blockIdx.x * 8 + warp, b = blockIdx.z;
  const int g0 = blockIdx.y * BC_GCH, g1 = min(G, g0 + BC_GCH);
  if (t >= Tn) return;
  const bool act = n0 < N;
  const size_t in_off = (size_t)(4 * g0 + 2 * which) * N + n0;
  const T* src = bc + ((size_t)b * Tn + t) * bcs + in_off;
  T* dst = dbc + ((size_t)b * Tn + t) * dbcs + in_off;
  const T* grad = (which ? dCo : dBo) + (((size_t)b * G + g0) * Tn + t) * 2 * N + 2 * n0;
  const size_t gstep = (size_t)Tn * 2 * N;
  const float inv_n = 1.f / (float)N;
  Raw4<T> na{}, np{};
  Raw8<T> ng{};
  auto fetch = [&] {
    if (!act) return;
    na = *reinterpret_cast<const Raw4<T>*>(src);
    np = *reinterpret_cast<const Raw4<T>*>(src + N);
    ng = load_raw8<T>(grad);
  };
  fetch();
#pragma unroll 2
  for (int g = g0; g < g1; ++g) {
    f2 xa[2], xp[2], gre[2], gim[2], a[2], th[2], sn[2], cs[2], dot[2];
    unpack4<T>(na, xa); unpack4<T>(np, xp);
    split8<T>(ng, gre, gim);
    src += 4 * N; grad += gstep;
    if (g + 1 < g1) fetch();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[i] = softplus2<FAST>(xa[i]);
      th[i] = tanh2<FAST>(xp[i]);
      sincos2<FAST>(mul2(th[i], dup2(3.14159265358979323846f)), &sn[i], &cs[i]);
      dot[i] = fma2(sn[i], gim[i], mul2(cs[i], gre[i]));
    }
    const float2 sq = un2(fma2(a[0], a[0], mul2(a[1], a[1]))), gs = un2(fma2(a[0], dot[0], mul2(a[1], dot[1])));
    const float ss = part_sum<WIDE>(act ? sq.x + sq.y : 0.f), gsum = part_sum<WIDE>(act ? gs.x + gs.y : 0.f);
    if (act) {
      const float ms = ss * inv_n, inv = rsqrtf(fmaxf(ms, eps));
      const f2 inv2 = dup2(inv), g_ms = dup2(ms > eps ? -inv * inv * inv * gsum * inv_n : 0.f);
      f2 da[2], dp[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const f2 g_amp = fma2(inv2, dot[i], mul2(g_ms, a[i]));
        da[i] = mul2(g_amp, sigmoid_pair<FAST>(xa[i]));
        const f2 cross = fma2(cs[i], gim[i], mul2(mul2(sn[i], gre[i]), dup2(-1.f)));
        const f2 slope = fma2(mul2(th[i], th[i]), dup2(-3.14159265358979323846f), dup2(3.14159265358979323846f));
        dp[i] = mul2(mul2(mul2(a[i], inv2), cross), slope);
      }
      store4<T>(dst, da);
      store4<T>(dst + N, dp);
    }
    dst += 4 * N;
  }
}

// (the logits and their gradients are read and written 4 at a time: 8 bytes of 16-bit values)
inline bool bc_vec_ok(int batch, int groups, int N, const void* a, const void* b, const void* c, const void* d, int64_t bcs,
                      int64_t dbcs, int io) {
  const size_t in = io == SL_F32 ? 16 : 8;
  return batch <= 65535 && (groups + BC_GCH - 1) / BC_GCH <= 65535 && N % 4 == 0 && N <= 128 && aligned(a, in) &&
         aligned(b, 16) && aligned(c, 16) && (d == nullptr || aligned(d, in)) && bcs % 4 == 0 && dbcs % 4 == 0;
}

// (the coefficient arithmetic - zc, CoeffOut, wrap_angle_f, coeff_eval - lives in scanprep_math.cuh)
struct CoeffParams {
  const void* params;
  const float *dt_bias, *alpha_bias, *theta_mod_bias, *theta_bias, *theta_sign;
  sl_scanprep_config cfg;
  float *M, *K;
  const float *dM, *dK;
  void* dparams;
  int64_t ps, dps;              // row strides of params and dparams
  float *d_dt_bias, *d_alpha_bias, *d_theta_mod_bias, *d_theta_bias;
  int batch, T, H;
};

// grid (ceil(T/128), H, batch), thread = token: outputs are coalesced along T.
template <typename T>
__global__ void __launch_bounds__(128) coeff_fwd_kernel(CoeffParams p) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, h = blockIdx.y, b = blockIdx.z;
  if (t >= p.T) return;
  const T* pr = reinterpret_cast<const T*>(p.params) + ((size_t)b * p.T + t) * p.ps + 3 * h;
  const CoeffOut o = coeff_eval<false>(to_f32(pr[0]) + p.dt_bias[h], to_f32(pr[1]) + p.alpha_bias[h],
                                to_f32(pr[2]) + p.theta_mod_bias[h], p.theta_bias[h],
                                p.theta_sign[h], p.cfg);
  const size_t i = ((size_t)b * p.H + h) * p.T + t;
  reinterpret_cast<float2*>(p.M)[i] = make_float2((float)o.rho.re, (float)o.rho.im);
  const zc kp = {o.dt * o.k2.re, o.dt * o.k2.im};
  const zc kc = {o.dt * o.k1.re - kp.re, o.dt * o.k1.im - kp.im};
  reinterpret_cast<float4*>(p.K)[i] = make_float4((float)kp.re, (float)kp.im, (float)kc.re, (float)kc.im);
}

template <typename T>
__global__ void __launch_bounds__(128) coeff_bwd_kernel(CoeffParams p) {
  __shared__ float s_red[4][4];
  const int t = blockIdx.x * blockDim.x + threadIdx.x, h = blockIdx.y, b = blockIdx.z;
  float g0 = 0.f, g1 = 0.f, g2 = 0.f, gx = 0.f;
  if (t < p.T) {
    const T* pr = reinterpret_cast<const T*>(p.params) + ((size_t)b * p.T + t) * p.ps + 3 * h;
    const CoeffOut o = coeff_eval(to_f32(pr[0]) + p.dt_bias[h], to_f32(pr[1]) + p.alpha_bias[h],
                                  to_f32(pr[2]) + p.theta_mod_bias[h], p.theta_bias[h],
                                  p.theta_sign[h], p.cfg);
    const size_t i = ((size_t)b * p.H + h) * p.T + t;
    const float2 gm = reinterpret_cast<const float2*>(p.dM)[i];
    const float4 gk = reinterpret_cast<const float4*>(p.dK)[i];
    const zc gM = {gm.x, gm.y}, gKp = {gk.x, gk.y}, gKc = {gk.z, gk.w};
    // kp = dt k2 ; kc = dt (k1 - k2)
    const zc gk1 = {o.dt * gKc.re, o.dt * gKc.im};
    const zc gk2 = {o.dt * (gKp.re - gKc.re), o.dt * (gKp.im - gKc.im)};
    const zc k12 = {o.k1.re - o.k2.re, o.k1.im - o.k2.im};
    const double g_dt = (o.k2.re * gKp.re + o.k2.im * gKp.im) + (k12.re * gKc.re + k12.im * gKc.im);
    zc gz = zconj_mul(o.rho, gM);
    const zc a1 = zconj_mul(o.dk1, gk1), a2 = zconj_mul(o.dk2, gk2);
    gz.re += a1.re + a2.re; gz.im += a1.im + a2.im;
    const double g_r = gz.re / o.r;
    const double g_alpha = -(double)(p.cfg.r_max - p.cfg.r_min) * o.ea * g_r;
    const double span = fmax((double)p.cfg.theta_init_max - (double)p.cfg.theta_init_min, 1.0e-6);
    const double g_thu = span * (double)p.theta_sign[h] * gz.im;
    const double g_x = o.dsg_thu * g_thu;
    g0 = (float)((double)(p.cfg.dt_max - p.cfg.dt_min) * o.dsg_dt * g_dt);
    g1 = (float)((double)(p.cfg.alpha_max - p.cfg.alpha_min) * o.dsg_al * g_alpha);
    g2 = (float)((double)p.cfg.theta_mod_scale * (1.0 - o.tanh2) * g_x);
    gx = (float)g_x;
    T* dp = reinterpret_cast<T*>(p.dparams) + ((size_t)b * p.T + t) * p.dps + 3 * h;
    dp[0] = from_f32<T>(g0); dp[1] = from_f32<T>(g1); dp[2] = from_f32<T>(g2);
  }
  g0 = warp_sum(g0); g1 = warp_sum(g1); g2 = warp_sum(g2); gx = warp_sum(gx);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { s_red[w][0] = g0; s_red[w][1] = g1; s_red[w][2] = g2; s_red[w][3] = gx; }
  __syncthreads();
  if (threadIdx.x < 4) {
    const float s = s_red[0][threadIdx.x] + s_red[1][threadIdx.x] + s_red[2][threadIdx.x] + s_red[3][threadIdx.x];
    float* dst = threadIdx.x == 0 ? p.d_dt_bias : threadIdx.x == 1 ? p.d_alpha_bias
                 : threadIdx.x == 2 ? p.d_theta_mod_bias : p.d_theta_bias;
    if (dst) atomicAdd(dst + h, s);
  }
}

int check_common(int batch, int heads, int groups, int T, int P, int N, int io_dtype, int d_conv) {
  if (batch < 1 || heads < 1 || groups < 1 || heads % groups || T < 1 || P < 1 || N < 1)
    return SL_ERR_BAD_SHAPE;
  if (d_conv < 1 || d_conv > 4) return SL_ERR_UNSUPPORTED;
  if (!dtype_ok(io_dtype)) return SL_ERR_UNSUPPORTED;
  return SL_OK;
}

// ---- the three parts of a call (value, B/C, coefficients) touch disjoint tensors -----------------------
// For sequence-sized calls they are launched on three streams between a fork and a join on the caller's
// stream: the B/C kernels are bound by instruction issue, the value kernels by latency, and each leaves most
// of the DRAM bandwidth idle, so they overlap well.  The side streams and events are created on the first
// such call of a device (do that call outside stream capture); fork and join are ordinary event
// dependencies, so a captured call records them as edges of the graph.  SLINOSS_B200_SERIAL_PARTS=1 keeps
// every part on the caller's stream.
struct PartStreams {
  cudaStream_t side[2];
  cudaEvent_t start, done[2];
  bool tried, ok;
  std::mutex in_use;   // held from fork to join: the events are shared by all calls on the device
};
PartStreams* part_streams() {
  static PartStreams table[16];
  static std::mutex guard;   // forward and backward may arrive from different host threads
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return nullptr;
  std::lock_guard<std::mutex> lock(guard);
  PartStreams& ps = table[dev];
  if (!ps.tried) {
    ps.tried = true;
    const char* e = getenv("SLINOSS_B200_SERIAL_PARTS");
    ps.ok = !(e && e[0] == '1');
    for (int i = 0; i < 2 && ps.ok; ++i)
      ps.ok = cudaStreamCreateWithFlags(&ps.side[i], cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreateWithFlags(&ps.done[i], cudaEventDisableTiming) == cudaSuccess;
    ps.ok = ps.ok && cudaEventCreateWithFlags(&ps.start, cudaEventDisableTiming) == cudaSuccess;
    if (!ps.ok) cudaGetLastError();
  }
  return ps.ok ? &ps : nullptr;
}
// Streams of the (value, B/C, coefficient) parts of one call; join() orders the caller's stream after all.
struct PartFork {
  cudaStream_t v, b, c;
  PartStreams* ps = nullptr;
  cudaStream_t main;
  ~PartFork() { join(); }
  PartFork(cudaStream_t st, int parts, long long rows) : v(st), b(st), c(st), main(st) {
    if (parts < 2 || rows < 2048) return;
    ps = part_streams();
    if (!ps) return;
    ps->in_use.lock();
    if (cudaEventRecord(ps->start, st) != cudaSuccess || cudaStreamWaitEvent(ps->side[0], ps->start, 0) != cudaSuccess ||
        cudaStreamWaitEvent(ps->side[1], ps->start, 0) != cudaSuccess) {
      cudaGetLastError();
      ps->in_use.unlock();
      ps = nullptr;
      return;
    }
    b = ps->side[0];
    c = ps->side[1];
  }
  void join() {
    if (!ps) return;
    for (int i = 0; i < 2; ++i) {
      cudaEventRecord(ps->done[i], ps->side[i]);
      cudaStreamWaitEvent(main, ps->done[i], 0);
    }
    ps->in_use.unlock();
    ps = nullptr;
  }
};

}  // namespace

int scanprep_fwd(const ScanPrepArgs& a, const ScanPrepOut& o, cudaStream_t st) {
  if (int e = check_common(a.batch, a.heads, a.groups, a.T, a.P, a.N, a.io_dtype, a.conv_weight ? a.d_conv : 1)) return e;
  if (a.value && !o.U) return SL_ERR_NULL_POINTER;
  if (a.bc && (!o.B || !o.C || !a.cfg)) return SL_ERR_NULL_POINTER;
  if (a.params) {
    if (!o.M || !o.K || !a.cfg || !a.dt_bias || !a.alpha_bias || !a.theta_mod_bias || !a.theta_bias || !a.theta_sign)
      return SL_ERR_NULL_POINTER;
    if (!aligned(o.M, 8) || !aligned(o.K, 16)) return SL_ERR_BAD_ALIGNMENT;
  }
  const int batch = a.batch, T = a.T, heads = a.heads, groups = a.groups, N = a.N;
  PartFork fork(st, (a.value != nullptr) + (a.bc != nullptr) + (a.params != nullptr), (long long)batch * T);
  if (a.value) {
    ValueParams p{};
    p.x = a.value; p.w = a.conv_weight; p.bias = a.conv_bias; p.state_in = a.conv_state_in;
    p.state_out = a.conv_state_out; p.U = o.U; p.xs = a.value_stride;
    p.usb = a.u_b; p.ush = a.u_h; p.ust = a.u_t;
    p.batch = batch; p.T = T; p.C = heads * a.P; p.P = a.P; p.W = a.conv_weight ? a.d_conv : 1;
    if (value_vec_ok(p, nullptr, nullptr)) {
      const int tile = conv_tile(T, p.C, batch);
      dim3 grid((p.C + 32 * CONV_V - 1) / (32 * CONV_V), (T + CONV_SUB * tile - 1) / (CONV_SUB * tile), batch);
      SL_DISPATCH_DTYPE(a.io_dtype, Tt, { value_fwd_vec_kernel<Tt><<<grid, 256, 0, fork.v>>>(p, tile); });
    } else {
      dim3 grid((p.C + 255) / 256, (T + CONV_TT - 1) / CONV_TT, batch);
      SL_DISPATCH_DTYPE(a.io_dtype, Tt, { value_fwd_kernel<Tt><<<grid, 256, 0, fork.v>>>(p); });
    }
    note_launches(1);
  }
  if (a.bc) {
    const long long rows = (long long)batch * T * groups;
    const bool wide = N > 64;
    const dim3 vgrid((T + (wide ? 3 : 7)) / (wide ? 4 : 8), (groups + BC_GCH - 1) / BC_GCH, batch);
    const float eps = a.cfg->eps;
    SL_DISPATCH_DTYPE(a.io_dtype, Tt, {
      const Tt* bc = reinterpret_cast<const Tt*>(a.bc);
      Tt *Bo = reinterpret_cast<Tt*>(o.B), *Co = reinterpret_cast<Tt*>(o.C);
      if (!bc_vec_ok(batch, groups, N, bc, Bo, Co, nullptr, a.bc_stride, 0, a.io_dtype))
        bc_fwd_kernel<Tt><<<(unsigned)((rows + 7) / 8), 256, 0, fork.b>>>(bc, Bo, Co, a.bc_stride, batch, T, groups, N, eps);
      else if (wide)
        bc_fwd_vec_kernel<Tt, true><<<vgrid, 256, 0, fork.b>>>(bc, Bo, Co, a.bc_stride, T, groups, N, eps);
      else
        bc_fwd_vec_kernel<Tt, false><<<vgrid, 256, 0, fork.b>>>(bc, Bo, Co, a.bc_stride, T, groups, N, eps);
    });
    note_launches(1);
  }
  if (a.params) {
    CoeffParams p{};
    p.params = a.params; p.ps = a.params_stride; p.dt_bias = a.dt_bias; p.alpha_bias = a.alpha_bias;
    p.theta_mod_bias = a.theta_mod_bias; p.theta_bias = a.theta_bias; p.theta_sign = a.theta_sign;
    p.cfg = *a.cfg; p.M = o.M; p.K = o.K; p.batch = batch; p.T = T; p.H = heads;
    dim3 grid((T + 127) / 128, heads, batch);
    SL_DISPATCH_DTYPE(a.io_dtype, Tt, { coeff_fwd_kernel<Tt><<<grid, 128, 0, fork.c>>>(p); });
    note_launches(1);
  }
  fork.join();
  return launch_status();
}

int scanprep_bwd(const ScanPrepArgs& a, const ScanPrepGrads& g, cudaStream_t st) {
  if (int e = check_common(a.batch, a.heads, a.groups, a.T, a.P, a.N, a.io_dtype, a.conv_weight ? a.d_conv : 1)) return e;
  if (g.dU && (!g.d_value || !a.value || (a.conv_weight && !g.d_conv_weight) || (g.dY && !g.skip))) return SL_ERR_NULL_POINTER;
  if (g.dB && (!g.dC || !a.bc || !g.d_bc || !a.cfg)) return SL_ERR_NULL_POINTER;
  if (g.dM) {
    if (!g.dK || !a.params || !g.d_params || !a.cfg || !a.dt_bias || !a.alpha_bias || !a.theta_mod_bias || !a.theta_bias ||
        !a.theta_sign)
      return SL_ERR_NULL_POINTER;
    if (!aligned(g.dM, 8) || !aligned(g.dK, 16)) return SL_ERR_BAD_ALIGNMENT;
  }
  const int batch = a.batch, T = a.T, heads = a.heads, groups = a.groups, N = a.N;
  PartFork fork(st, (g.dU != nullptr) + (g.dB != nullptr) + (g.dM != nullptr), (long long)batch * T);
  if (g.dU) {
    ValueBwdParams q{};
    ValueParams& p = q.f;
    p.x = a.value; p.w = a.conv_weight; p.bias = a.conv_bias; p.state_in = a.conv_state_in;
    p.xs = a.value_stride; p.usb = a.u_b; p.ush = a.u_h; p.ust = a.u_t;
    p.batch = batch; p.T = T; p.C = heads * a.P; p.P = a.P; p.W = a.conv_weight ? a.d_conv : 1;
    q.dU = g.dU; q.dx = g.d_value; q.dxs = g.d_value_stride; q.dstate = g.d_conv_state; q.dw = g.d_conv_weight;
    q.dbias = g.d_conv_bias; q.dY = g.dY; q.skip = g.skip;
    ValueParams pv = p;
    pv.U = const_cast<void*>(g.dU);
    if (value_vec_ok(pv, g.d_value, nullptr) && g.d_value_stride % CONV_V == 0 && aligned(g.dY, 16)) {
      const int tile = conv_tile(T, p.C, batch);
      dim3 grid((p.C + 32 * CONV_V - 1) / (32 * CONV_V), (T + CONV_SUB * tile - 1) / (CONV_SUB * tile), batch);
      SL_DISPATCH_DTYPE(a.io_dtype, Tt, {
        if (g.dY) value_bwd_vec_kernel<Tt, true><<<grid, 256, 0, fork.v>>>(q, tile);
        else value_bwd_vec_kernel<Tt, false><<<grid, 256, 0, fork.v>>>(q, tile);
      });
    } else {
      dim3 grid((p.C + 255) / 256, (T + CONV_TT - 1) / CONV_TT, batch);
      SL_DISPATCH_DTYPE(a.io_dtype, Tt, { value_bwd_kernel<Tt><<<grid, 256, 0, fork.v>>>(q); });
    }
    note_launches(1);
  }
  if (g.dB) {
    const long long rows = (long long)batch * T * groups;
    const bool wide = N > 64;
    const dim3 vgrid((T + (wide ? 3 : 7)) / (wide ? 4 : 8), (groups + BC_GCH - 1) / BC_GCH, batch);
    const float eps = a.cfg->eps;
    SL_DISPATCH_DTYPE(a.io_dtype, Tt, {
      const Tt *bc = reinterpret_cast<const Tt*>(a.bc), *dB = reinterpret_cast<const Tt*>(g.dB);
      const Tt* dC = reinterpret_cast<const Tt*>(g.dC);
      Tt* dbc = reinterpret_cast<Tt*>(g.d_bc);
      if (!bc_vec_ok(batch, groups, N, bc, dB, dC, dbc, a.bc_stride, g.d_bc_stride, a.io_dtype))
        bc_bwd_kernel<Tt><<<(unsigned)((rows + 7) / 8), 256, 0, fork.b>>>(bc, dB, dC, dbc, a.bc_stride, g.d_bc_stride, batch, T,
                                                                          groups, N, eps);
      else if (wide)
        bc_bwd_vec_kernel<Tt, true><<<vgrid, 256, 0, fork.b>>>(bc, dB, dC, dbc, a.bc_stride, g.d_bc_stride, T, groups, N, eps);
      else
        bc_bwd_vec_kernel<Tt, false><<<vgrid, 256, 0, fork.b>>>(bc, dB, dC, dbc, a.bc_stride, g.d_bc_stride, T, groups, N, eps);
    });
    note_launches(1);
  }
  if (g.dM) {
    CoeffParams p{};
    p.params = a.params; p.ps = a.params_stride; p.dt_bias = a.dt_bias; p.alpha_bias = a.alpha_bias;
    p.theta_mod_bias = a.theta_mod_bias; p.theta_bias = a.theta_bias; p.theta_sign = a.theta_sign;
    p.cfg = *a.cfg; p.dM = g.dM; p.dK = g.dK; p.dparams = g.d_params; p.dps = g.d_params_stride; p.d_dt_bias = g.d_dt_bias;
    p.d_alpha_bias = g.d_alpha_bias; p.d_theta_mod_bias = g.d_theta_mod_bias;
    p.d_theta_bias = g.d_theta_bias; p.batch = batch; p.T = T; p.H = heads;
    dim3 grid((T + 127) / 128, heads, batch);
    SL_DISPATCH_DTYPE(a.io_dtype, Tt, { coeff_bwd_kernel<Tt><<<grid, 128, 0, fork.c>>>(p); });
    note_launches(1);
  }
  fork.join();
  return launch_status();
}

}  // namespace sl

extern "C" int sl_scanprep_conv_fwd(const void* value, int64_t value_row_stride,
                                    const void* conv_weight, const void* conv_bias,
                                    const void* conv_state_in, void* conv_state_out, int d_conv,
                                    const void* params, const void* bc, const float* dt_bias,
                                    const float* alpha_bias, const float* theta_mod_bias,
                                    const float* theta_bias, const float* theta_sign,
                                    const sl_scanprep_config* cfg, void* U, int64_t u_stride_b,
                                    int64_t u_stride_h, int64_t u_stride_t, float* M, float* K,
                                    void* Bo, void* Co, int batch, int heads, int groups, int T,
                                    int P, int N, int io_dtype, void* stream) {
  const sl::ScanPrepArgs a{value, value_row_stride, conv_weight, conv_bias, conv_state_in, conv_state_out, d_conv,
                           params, 3 * (int64_t)heads, bc, 4 * (int64_t)groups * N, dt_bias, alpha_bias, theta_mod_bias,
                           theta_bias, theta_sign, cfg, u_stride_b, u_stride_h, u_stride_t, batch, heads, groups, T, P, N,
                           io_dtype};
  return sl::scanprep_fwd(a, sl::ScanPrepOut{U, M, K, Bo, Co}, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int sl_scanprep_conv_bwd(
    const void* value, int64_t value_row_stride, const void* conv_weight, const void* conv_bias,
    const void* conv_state_in, int d_conv, const void* params, const void* bc,
    const float* dt_bias, const float* alpha_bias, const float* theta_mod_bias,
    const float* theta_bias, const float* theta_sign, const sl_scanprep_config* cfg,
    const void* dU, int64_t u_stride_b, int64_t u_stride_h, int64_t u_stride_t, const float* dM,
    const float* dK, const void* dBo, const void* dCo, void* d_value, float* d_conv_weight,
    float* d_conv_bias, void* d_conv_state, void* d_params, void* d_bc, float* d_dt_bias,
    float* d_alpha_bias, float* d_theta_mod_bias, float* d_theta_bias, int batch, int heads,
    int groups, int T, int P, int N, int io_dtype, void* stream) {
  const int64_t params_row = 3 * (int64_t)heads, bc_row = 4 * (int64_t)groups * N;
  const sl::ScanPrepArgs a{value, value_row_stride, conv_weight, conv_bias, conv_state_in, nullptr, d_conv, params, params_row,
                           bc, bc_row, dt_bias, alpha_bias, theta_mod_bias, theta_bias, theta_sign, cfg, u_stride_b, u_stride_h,
                           u_stride_t, batch, heads, groups, T, P, N, io_dtype};
  const sl::ScanPrepGrads g{dU, dM, dK, dBo, dCo, d_value, (int64_t)heads * P, d_conv_weight, d_conv_bias, d_conv_state, d_params,
                            params_row, d_bc, bc_row, d_dt_bias, d_alpha_bias, d_theta_mod_bias, d_theta_bias};
  return sl::scanprep_bwd(a, g, reinterpret_cast<cudaStream_t>(stream));
}
