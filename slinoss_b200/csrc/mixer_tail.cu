// Row-wise part of the mixer tail: skip connection, SiLU gate and RMSNorm.
//
//   pre    = Y + d_skip[h] * U                 (float32, rounded to the io dtype)
//   hidden = pre * SiLU(gate)                  (float32, rounded to the io dtype)
//   normed = hidden * rsqrt(mean(hidden^2) + eps) * w
//
// Reference: slinoss/ops/mixer/tail.py:63-142 (the roundings above are the ones
// the reference makes between its steps).  One CTA owns one (batch, token) row of
// heads*P channels; Y and U are read in their (batch, heads, T, P) layout and the
// result is written channel-last, ready for the out_proj GEMM.
#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

constexpr int TAIL_THREADS = 256;
constexpr int TAIL_MAX_PER_THREAD = 16;  // channels <= 4096

template <typename T>
__device__ __forceinline__ float round_io(float v) { return to_f32(from_f32<T>(v)); }

__device__ __forceinline__ float block_sum(float v, float* s_red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) s_red[w] = v;
  __syncthreads();
  float s = 0.f;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += s_red[k];
  return s;
}

struct TailParams {
  const void *Y, *gate, *skip, *w, *dn;
  const float* d_skip;
  void *normed, *dY, *dgate, *dskip_in;
  float *d_d_skip, *d_w;
  int64_t gs, dgs;   // row strides of gate and dgate
  float eps;
  int batch, H, T, P;
};

template <typename T>
__global__ void __launch_bounds__(TAIL_THREADS) tail_fwd_kernel(TailParams p) {
  __shared__ float s_red[TAIL_THREADS / 32];
  const int C = p.H * p.P;
  const T* Y = reinterpret_cast<const T*>(p.Y);
  const T* S = reinterpret_cast<const T*>(p.skip);
  const T* gate = reinterpret_cast<const T*>(p.gate);
  const T* w = reinterpret_cast<const T*>(p.w);
  T* out = reinterpret_cast<T*>(p.normed);
  for (long long row = blockIdx.x; row < (long long)p.batch * p.T; row += gridDim.x) {
    const int t = (int)(row % p.T), b = (int)(row / p.T);
    float hid[TAIL_MAX_PER_THREAD];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) {
      const int c = threadIdx.x + i * TAIL_THREADS;
      hid[i] = 0.f;
      if (c < C) {
        const int h = c / p.P, pp = c - h * p.P;
        const size_t yi = (((size_t)b * p.H + h) * p.T + t) * p.P + pp;
        float pre = to_f32(Y[yi]);
        if (S) pre = round_io<T>(pre + to_f32(S[yi]) * p.d_skip[h]);
        const float g = to_f32(gate[(size_t)row * p.gs + c]);
        hid[i] = round_io<T>(pre * silu_f(g));
        ss += hid[i] * hid[i];
      }
    }
    ss = block_sum(ss, s_red);
    const float rstd = rsqrtf(ss / (float)C + p.eps);
#pragma unroll
    for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) {
      const int c = threadIdx.x + i * TAIL_THREADS;
      if (c < C) out[(size_t)row * C + c] = from_f32<T>(hid[i] * rstd * to_f32(w[c]));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(TAIL_THREADS) tail_bwd_kernel(TailParams p) {
  __shared__ float s_red[TAIL_THREADS / 32];
  extern __shared__ float s_dskip[];  // H floats
  const int C = p.H * p.P;
  const T* Y = reinterpret_cast<const T*>(p.Y);
  const T* S = reinterpret_cast<const T*>(p.skip);
  const T* gate = reinterpret_cast<const T*>(p.gate);
  const T* w = reinterpret_cast<const T*>(p.w);
  const T* dn = reinterpret_cast<const T*>(p.dn);
  T* dY = reinterpret_cast<T*>(p.dY);
  T* dgate = reinterpret_cast<T*>(p.dgate);
  T* dS = reinterpret_cast<T*>(p.dskip_in);
  float dw_acc[TAIL_MAX_PER_THREAD];
#pragma unroll
  for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) dw_acc[i] = 0.f;
  for (int i = threadIdx.x; i < p.H; i += blockDim.x) s_dskip[i] = 0.f;
  __syncthreads();
  for (long long row = blockIdx.x; row < (long long)p.batch * p.T; row += gridDim.x) {
    const int t = (int)(row % p.T), b = (int)(row / p.T);
    float hid[TAIL_MAX_PER_THREAD], gw[TAIL_MAX_PER_THREAD];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) {
      const int c = threadIdx.x + i * TAIL_THREADS;
      hid[i] = gw[i] = 0.f;
      if (c < C) {
        const int h = c / p.P, pp = c - h * p.P;
        const size_t yi = (((size_t)b * p.H + h) * p.T + t) * p.P + pp;
        float pre = to_f32(Y[yi]);
        if (S) pre = round_io<T>(pre + to_f32(S[yi]) * p.d_skip[h]);
        const float g = to_f32(gate[(size_t)row * p.gs + c]);
        hid[i] = round_io<T>(pre * silu_f(g));
        gw[i] = to_f32(dn[(size_t)row * C + c]) * to_f32(w[c]);
        ss += hid[i] * hid[i];
        dot += hid[i] * gw[i];
      }
    }
    ss = block_sum(ss, s_red);
    dot = block_sum(dot, s_red);
    const float rstd = rsqrtf(ss / (float)C + p.eps);
    const float coef = dot * rstd * rstd * rstd / (float)C;
#pragma unroll
    for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) {
      const int c = threadIdx.x + i * TAIL_THREADS;
      if (c < C) {
        const int h = c / p.P, pp = c - h * p.P;
        const size_t yi = (((size_t)b * p.H + h) * p.T + t) * p.P + pp;
        const float dnv = to_f32(dn[(size_t)row * C + c]);
        dw_acc[i] += dnv * hid[i] * rstd;
        const float dh = rstd * gw[i] - hid[i] * coef;
        float pre = to_f32(Y[yi]);
        float sv = 0.f;
        if (S) { sv = to_f32(S[yi]); pre = round_io<T>(pre + sv * p.d_skip[h]); }
        const float g = to_f32(gate[(size_t)row * p.gs + c]);
        const float sg = sigmoid_f(g);
        const float dpre = dh * g * sg;
        dgate[(size_t)row * p.dgs + c] = from_f32<T>(dh * pre * sg * (1.f + g * (1.f - sg)));
        dY[yi] = from_f32<T>(dpre);
        if (S) {
          if (dS) dS[yi] = from_f32<T>(dpre * p.d_skip[h]);
          atomicAdd(&s_dskip[h], dpre * sv);
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TAIL_MAX_PER_THREAD; ++i) {
    const int c = threadIdx.x + i * TAIL_THREADS;
    if (c < C) atomicAdd(p.d_w + c, dw_acc[i]);
  }
  if (S && p.d_d_skip)
    for (int i = threadIdx.x; i < p.H; i += blockDim.x) atomicAdd(p.d_d_skip + i, s_dskip[i]);
}

// ---- vector path: every thread owns 16-byte pieces (8 or 4 channels of one head) ---------------
// Needs P % V == 0 (a piece never straddles two heads), 16-byte aligned pointers and a gate row
// stride that is a multiple of V.  One CTA owns one row at a time; a thread keeps the same
// channels for every row it visits, so the weight / skip gradients are accumulated in registers
// over the CTA's rows and added to the float32 accumulators once at the end.
constexpr int TAIL_VIT_MAX = 2;   // pieces per thread: channels <= 2 * 256 * V

template <typename T, int TAIL_VIT>
__global__ void __launch_bounds__(TAIL_THREADS) tail_fwd_vec_kernel(TailParams p) {
  constexpr int V = Vec16<T>::N;
  __shared__ float s_red[TAIL_THREADS / 32];
  const int C = p.H * p.P;
  const T* Y = reinterpret_cast<const T*>(p.Y);
  const T* S = reinterpret_cast<const T*>(p.skip);
  const T* gate = reinterpret_cast<const T*>(p.gate);
  const T* w = reinterpret_cast<const T*>(p.w);
  T* out = reinterpret_cast<T*>(p.normed);
  float wv[TAIL_VIT][V], dsk[TAIL_VIT];
  int hh[TAIL_VIT], pp[TAIL_VIT];
#pragma unroll
  for (int i = 0; i < TAIL_VIT; ++i) {
    const int c = (threadIdx.x + i * TAIL_THREADS) * V;
    hh[i] = 0; pp[i] = 0; dsk[i] = 0.f;
    if (c < C) {
      hh[i] = c / p.P; pp[i] = c - hh[i] * p.P;
      load16<T>(w + c, wv[i]);
      if (S) dsk[i] = p.d_skip[hh[i]];
    }
  }
  // The raw 16-byte pieces of the NEXT row are fetched before the current row is reduced, so the
  // loads overlap the block reduction and the stores.
  const unsigned rows = (unsigned)p.batch * (unsigned)p.T;   // < 2^31, checked by the launcher
  uint4 nY[TAIL_VIT], nG[TAIL_VIT], nS[TAIL_VIT];
  auto fetch = [&](unsigned row) {
    const int t = (int)(row % (unsigned)p.T), b = (int)(row / (unsigned)p.T);
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        const size_t yi = (((size_t)b * p.H + hh[i]) * p.T + t) * p.P + pp[i];
        nY[i] = *reinterpret_cast<const uint4*>(Y + yi);
        nG[i] = *reinterpret_cast<const uint4*>(gate + (size_t)row * p.gs + c);
        if (S) nS[i] = *reinterpret_cast<const uint4*>(S + yi);
      }
    }
  };
  if (blockIdx.x < rows) fetch(blockIdx.x);
  for (unsigned row = blockIdx.x; row < rows; row += gridDim.x) {
    uint4 cY[TAIL_VIT], cG[TAIL_VIT], cS[TAIL_VIT];
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) { cY[i] = nY[i]; cG[i] = nG[i]; cS[i] = nS[i]; }
    if (row + gridDim.x < rows) fetch(row + gridDim.x);
    float hid[TAIL_VIT][V];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        float y[V], g[V];
        unpack16<T>(cY[i], y);
        unpack16<T>(cG[i], g);
        if (S) {
          float sv[V];
          unpack16<T>(cS[i], sv);
#pragma unroll
          for (int k = 0; k < V; k += 2) {
            y[k] += sv[k] * dsk[i]; y[k + 1] += sv[k + 1] * dsk[i];
            round_pair<T>(y[k], y[k + 1]);
          }
        }
#pragma unroll
        for (int k = 0; k < V; k += 2) {
          hid[i][k] = y[k] * silu_f(g[k]); hid[i][k + 1] = y[k + 1] * silu_f(g[k + 1]);
          round_pair<T>(hid[i][k], hid[i][k + 1]);
          ss += hid[i][k] * hid[i][k] + hid[i][k + 1] * hid[i][k + 1];
        }
      }
    }
    ss = block_sum(ss, s_red);
    const float rstd = rsqrtf(ss / (float)C + p.eps);
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        float o[V];
#pragma unroll
        for (int k = 0; k < V; ++k) o[k] = hid[i][k] * rstd * wv[i][k];
        store16<T>(out + (size_t)row * C + c, o);
      }
    }
  }
}

template <typename T, int TAIL_VIT>
__global__ void __launch_bounds__(TAIL_THREADS) tail_bwd_vec_kernel(TailParams p) {
  constexpr int V = Vec16<T>::N;
  __shared__ float s_red[TAIL_THREADS / 32];
  const int C = p.H * p.P;
  const T* Y = reinterpret_cast<const T*>(p.Y);
  const T* S = reinterpret_cast<const T*>(p.skip);
  const T* gate = reinterpret_cast<const T*>(p.gate);
  const T* w = reinterpret_cast<const T*>(p.w);
  const T* dn = reinterpret_cast<const T*>(p.dn);
  T* dY = reinterpret_cast<T*>(p.dY);
  T* dgate = reinterpret_cast<T*>(p.dgate);
  T* dS = reinterpret_cast<T*>(p.dskip_in);
  float wv[TAIL_VIT][V], dw_acc[TAIL_VIT][V], dsk[TAIL_VIT], dsk_acc[TAIL_VIT];
  int hh[TAIL_VIT], pp[TAIL_VIT];
#pragma unroll
  for (int i = 0; i < TAIL_VIT; ++i) {
    const int c = (threadIdx.x + i * TAIL_THREADS) * V;
    hh[i] = 0; pp[i] = 0; dsk[i] = 0.f; dsk_acc[i] = 0.f;
#pragma unroll
    for (int k = 0; k < V; ++k) dw_acc[i][k] = 0.f;
    if (c < C) {
      hh[i] = c / p.P; pp[i] = c - hh[i] * p.P;
      load16<T>(w + c, wv[i]);
      if (S) dsk[i] = p.d_skip[hh[i]];
    }
  }
  const unsigned rows = (unsigned)p.batch * (unsigned)p.T;   // < 2^31, checked by the launcher
  uint4 nY[TAIL_VIT], nG[TAIL_VIT], nS[TAIL_VIT], nD[TAIL_VIT];
  auto fetch = [&](unsigned row) {   // raw pieces of the next row, in flight while this one is reduced
    const int t = (int)(row % (unsigned)p.T), b = (int)(row / (unsigned)p.T);
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        const size_t yi = (((size_t)b * p.H + hh[i]) * p.T + t) * p.P + pp[i];
        nY[i] = *reinterpret_cast<const uint4*>(Y + yi);
        nG[i] = *reinterpret_cast<const uint4*>(gate + (size_t)row * p.gs + c);
        nD[i] = *reinterpret_cast<const uint4*>(dn + (size_t)row * C + c);
        if (S) nS[i] = *reinterpret_cast<const uint4*>(S + yi);
      }
    }
  };
  if (blockIdx.x < rows) fetch(blockIdx.x);
  for (unsigned row = blockIdx.x; row < rows; row += gridDim.x) {
    const int t = (int)(row % (unsigned)p.T), b = (int)(row / (unsigned)p.T);
    float pre[TAIL_VIT][V], sv[TAIL_VIT][V], g[TAIL_VIT][V], dnv[TAIL_VIT][V];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        unpack16<T>(nY[i], pre[i]);
        unpack16<T>(nG[i], g[i]);
        unpack16<T>(nD[i], dnv[i]);
        if (S) unpack16<T>(nS[i], sv[i]);
      }
    }
    if (row + gridDim.x < rows) fetch(row + gridDim.x);
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        if (S) {
#pragma unroll
          for (int k = 0; k < V; k += 2) {
            pre[i][k] += sv[i][k] * dsk[i]; pre[i][k + 1] += sv[i][k + 1] * dsk[i];
            round_pair<T>(pre[i][k], pre[i][k + 1]);
          }
        }
#pragma unroll
        for (int k = 0; k < V; k += 2) {
          float h0 = pre[i][k] * silu_f(g[i][k]), h1 = pre[i][k + 1] * silu_f(g[i][k + 1]);
          round_pair<T>(h0, h1);
          ss += h0 * h0 + h1 * h1;
          dot += h0 * dnv[i][k] * wv[i][k] + h1 * dnv[i][k + 1] * wv[i][k + 1];
        }
      }
    }
    ss = block_sum(ss, s_red);
    dot = block_sum(dot, s_red);
    const float rstd = rsqrtf(ss / (float)C + p.eps);
    const float coef = dot * rstd * rstd * rstd / (float)C;
#pragma unroll
    for (int i = 0; i < TAIL_VIT; ++i) {
      const int c = (threadIdx.x + i * TAIL_THREADS) * V;
      if (c < C) {
        const size_t yi = (((size_t)b * p.H + hh[i]) * p.T + t) * p.P + pp[i];
        float o_dy[V], o_dg[V], o_ds[V];
#pragma unroll
        for (int k2 = 0; k2 < V; k2 += 2) {
          float sgv[2], hidv[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            sgv[q] = sigmoid_f(g[i][k2 + q]);
            hidv[q] = pre[i][k2 + q] * (g[i][k2 + q] * sgv[q]);
          }
          round_pair<T>(hidv[0], hidv[1]);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int k = k2 + q;
            const float gg = g[i][k], sg = sgv[q], hid = hidv[q];
            dw_acc[i][k] += dnv[i][k] * hid * rstd;
            const float dh = rstd * dnv[i][k] * wv[i][k] - hid * coef;
            const float dpre = dh * gg * sg;
            o_dg[k] = dh * pre[i][k] * sg * (1.f + gg * (1.f - sg));
            o_dy[k] = dpre;
            if (S) { o_ds[k] = dpre * dsk[i]; dsk_acc[i] += dpre * sv[i][k]; }
          }
        }
        store16<T>(dgate + (size_t)row * p.dgs + c, o_dg);
        store16<T>(dY + yi, o_dy);
        if (S && dS) store16<T>(dS + yi, o_ds);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TAIL_VIT; ++i) {
    const int c = (threadIdx.x + i * TAIL_THREADS) * V;
    if (c < C) {
#pragma unroll
      for (int k = 0; k < V; ++k) atomicAdd(p.d_w + c + k, dw_acc[i][k]);
      if (S && p.d_d_skip) atomicAdd(p.d_d_skip + hh[i], dsk_acc[i]);
    }
  }
}

// Pair k of a 16-byte piece, and a pair put (rounded) into it.
template <typename T> __device__ __forceinline__ f2 pair_of(const uint4& r, int k) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
  if constexpr (sizeof(T) == 2) {
    const float2 q = unpack_pair<T>(w[k]);
    return mk2(q.x, q.y);
  } else {
    return mk2(__uint_as_float(w[2 * k]), __uint_as_float(w[2 * k + 1]));
  }
}
template <typename T> __device__ __forceinline__ void put_pair(uint32_t (&w)[4], int k, f2 v) {
  const float2 q = un2(v);
  if constexpr (sizeof(T) == 2) w[k] = pack_pair<T>(q.x, q.y);
  else { w[2 * k] = __float_as_uint(q.x); w[2 * k + 1] = __float_as_uint(q.y); }
}
__device__ __forceinline__ uint4 piece(const uint32_t (&w)[4]) { return make_uint4(w[0], w[1], w[2], w[3]); }

// The common width (heads * P <= 256 pieces of 16 bytes: one piece per thread) with fewer live registers, so that three
// CTAs stay resident per SM: between the two halves of a row its pieces stay packed, among them ``pre`` and ``hid``, which are
// rounded to the io type anyway; both row sums travel in one reduction, and its shared-memory slots alternate with the row so
// that one barrier per row is enough.  Was bound by instruction issue: 92 per channel, about 30 in packed pairs (16384 x 2048: 124 -> 110 us).  The CTA has just the warps the
// row fills: with a fixed 256 threads a row of 1152 channels left 44 % of the lanes idle.
template <typename T>
__global__ void __launch_bounds__(TAIL_THREADS, 3) tail_bwd_row_kernel(TailParams p) {
  constexpr int V = Vec16<T>::N;
  __shared__ float2 s_red[2][TAIL_THREADS / 32];
  const int C = p.H * p.P;
  const T* Y = reinterpret_cast<const T*>(p.Y);
  const T* S = reinterpret_cast<const T*>(p.skip);
  const T* gate = reinterpret_cast<const T*>(p.gate);
  const T* dn = reinterpret_cast<const T*>(p.dn);
  T* dY = reinterpret_cast<T*>(p.dY);
  T* dgate = reinterpret_cast<T*>(p.dgate);
  T* dS = reinterpret_cast<T*>(p.dskip_in);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = threadIdx.x * V;
  const bool act = c < C;
  const int hh = act ? c / p.P : 0, pp = c - hh * p.P;
  const float dsk = (act && S) ? p.d_skip[hh] : 0.f;
  uint4 wraw = make_uint4(0, 0, 0, 0);
  if (act) wraw = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.w) + c);
  f2 dw_acc[V / 2], dsk_acc = 0;
#pragma unroll
  for (int k = 0; k < V / 2; ++k) dw_acc[k] = 0;
  const unsigned rows = (unsigned)p.batch * (unsigned)p.T;   // < 2^31, checked by the launcher
  const size_t head_off = (size_t)hh * p.T * p.P + pp, batch_step = (size_t)p.H * p.T * p.P;
  uint4 nY = make_uint4(0, 0, 0, 0), nG = nY, nS = nY, nD = nY;
  auto fetch = [&](unsigned row) {
    if (!act) return;
    const unsigned b = row / (unsigned)p.T, t = row - b * (unsigned)p.T;
    const size_t yi = b * batch_step + head_off + (size_t)t * p.P;
    nY = *reinterpret_cast<const uint4*>(Y + yi);
    nG = *reinterpret_cast<const uint4*>(gate + (size_t)row * p.gs + c);
    nD = *reinterpret_cast<const uint4*>(dn + (size_t)row * C + c);
    if (S) nS = *reinterpret_cast<const uint4*>(S + yi);
  };
  if (blockIdx.x < rows) fetch(blockIdx.x);
  int par = 0;
  for (unsigned row = blockIdx.x; row < rows; row += gridDim.x, par ^= 1) {
    const uint4 cY = nY, cG = nG, cS = nS, cD = nD;
    if (row + gridDim.x < rows) fetch(row + gridDim.x);
    float ss = 0.f, dot = 0.f;
    uint32_t pre[4] = {cY.x, cY.y, cY.z, cY.w}, hid[4] = {0, 0, 0, 0};
    if (act) {
      f2 ss2 = 0, dot2 = 0;
#pragma unroll
      for (int k = 0; k < V / 2; ++k) {
        const f2 g = pair_of<T>(cG, k);
        if (S) put_pair<T>(pre, k, fma2(pair_of<T>(cS, k), dup2(dsk), pair_of<T>(cY, k)));
        put_pair<T>(hid, k, mul2(pair_of<T>(piece(pre), k), mul2(g, sigmoid2(g))));
        const f2 h = pair_of<T>(piece(hid), k);
        ss2 = fma2(h, h, ss2);
        dot2 = fma2(h, mul2(pair_of<T>(cD, k), pair_of<T>(wraw, k)), dot2);
      }
      const float2 a = un2(ss2), d = un2(dot2);
      ss = a.x + a.y; dot = d.x + d.y;
    }
    ss = warp_sum(ss); dot = warp_sum(dot);
    if (lane == 0) s_red[par][warp] = make_float2(ss, dot);
    __syncthreads();
    ss = 0.f; dot = 0.f;
#pragma unroll
    for (int k = 0; k < TAIL_THREADS / 32; ++k)
      if (k < (int)(blockDim.x >> 5)) { const float2 v = s_red[par][k]; ss += v.x; dot += v.y; }
    const float rstd = rsqrtf(ss / (float)C + p.eps);
    const float coef = dot * rstd * rstd * rstd / (float)C;
    if (act) {
      const unsigned b = row / (unsigned)p.T, t = row - b * (unsigned)p.T;
      const size_t yi = b * batch_step + head_off + (size_t)t * p.P;
      const f2 r2 = dup2(rstd), c2 = dup2(-coef);
      uint32_t o_dy[4], o_dg[4], o_ds[4];
#pragma unroll
      for (int k = 0; k < V / 2; ++k) {
        const f2 h = pair_of<T>(piece(hid), k), dnk = pair_of<T>(cD, k), g = pair_of<T>(cG, k), sg = sigmoid2(g);
        dw_acc[k] = fma2(dnk, mul2(h, r2), dw_acc[k]);
        const f2 dh = fma2(mul2(dnk, pair_of<T>(wraw, k)), r2, mul2(h, c2));
        const f2 silu = mul2(g, sg), dpre = mul2(dh, silu);
        put_pair<T>(o_dg, k, mul2(mul2(dh, pair_of<T>(piece(pre), k)), fma2(silu, fma2(sg, dup2(-1.f), dup2(1.f)), sg)));
        put_pair<T>(o_dy, k, dpre);
        if (S) {
          dsk_acc = fma2(dpre, pair_of<T>(cS, k), dsk_acc);
          if (dS) put_pair<T>(o_ds, k, mul2(dpre, dup2(dsk)));
        }
      }
      *reinterpret_cast<uint4*>(dgate + (size_t)row * p.dgs + c) = piece(o_dg);
      *reinterpret_cast<uint4*>(dY + yi) = piece(o_dy);
      if (S && dS) *reinterpret_cast<uint4*>(dS + yi) = piece(o_ds);
    }
  }
  // One atomic of the CTA per 4 weights and per head: adds to one 32-byte sector are serial in L2, and with one per thread
  // and weight the last wave of CTAs spent more on them than on its rows (figures at the launch).
  if (act) {
    if ((reinterpret_cast<uintptr_t>(p.d_w) & 15) == 0) {
#pragma unroll
      for (int k = 0; k < V; k += 4) {
        const float2 a = un2(dw_acc[k / 2]), b = un2(dw_acc[k / 2 + 1]);
        atomicAdd(reinterpret_cast<float4*>(p.d_w + c + k), make_float4(a.x, a.y, b.x, b.y));
      }
    } else {
#pragma unroll
      for (int k = 0; k < V / 2; ++k) {
        const float2 a = un2(dw_acc[k]);
        atomicAdd(p.d_w + c + 2 * k, a.x); atomicAdd(p.d_w + c + 2 * k + 1, a.y);
      }
    }
  }
  if (S && p.d_d_skip) {
    const int per_head = p.P / V;   // threads of one head
    const float2 both = un2(dsk_acc);
    float sum = both.x + both.y;
    if (per_head <= 32 && (per_head & (per_head - 1)) == 0) {   // whole warps, or an aligned share of one
      for (int o = per_head >> 1; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (act && (threadIdx.x & (per_head - 1)) == 0) atomicAdd(p.d_d_skip + hh, sum);
    } else if (act) {
      atomicAdd(p.d_d_skip + hh, sum);
    }
  }
}

template <typename T>
bool tail_vec_ok(const TailParams& p) {
  constexpr int V = Vec16<T>::N;
  const long long C = (long long)p.H * p.P;
  auto al = [](const void* q) { return q == nullptr || aligned(q, 16); };
  return (long long)p.batch * p.T < (1ll << 31) && p.P % V == 0 && p.gs % V == 0 && C <= (long long)TAIL_VIT_MAX * TAIL_THREADS * V && al(p.Y) &&
         al(p.gate) && al(p.skip) && al(p.w) && al(p.dn) && al(p.normed) && al(p.dY) && al(p.dgate) && p.dgs % V == 0 &&
         al(p.dskip_in);
}

int tail_check(const void* Y, const void* gate, const void* skip, const float* d_skip,
               const void* w, int batch, int heads, int T, int P, int io_dtype) {
  if (!Y || !gate || !w) return SL_ERR_NULL_POINTER;
  if ((skip == nullptr) != (d_skip == nullptr)) return SL_ERR_NULL_POINTER;
  if (batch < 1 || heads < 1 || T < 1 || P < 1) return SL_ERR_BAD_SHAPE;
  if ((long long)heads * P > (long long)TAIL_THREADS * TAIL_MAX_PER_THREAD) return SL_ERR_UNSUPPORTED;
  if (!dtype_ok(io_dtype)) return SL_ERR_UNSUPPORTED;
  return SL_OK;
}

}  // namespace
}  // namespace sl

extern "C" int sl_mixer_tail_fwd(const void* Y, const void* gate, int64_t gate_row_stride,
                                 const void* skip, const float* d_skip, const void* norm_weight,
                                 float eps, void* normed, int batch, int heads, int T, int P,
                                 int io_dtype, void* stream) {
  using namespace sl;
  if (int e = tail_check(Y, gate, skip, d_skip, norm_weight, batch, heads, T, P, io_dtype)) return e;
  if (!normed) return SL_ERR_NULL_POINTER;
  TailParams p{};
  p.Y = Y; p.gate = gate; p.skip = skip; p.w = norm_weight; p.d_skip = d_skip; p.normed = normed;
  p.gs = gate_row_stride; p.eps = eps; p.batch = batch; p.H = heads; p.T = T; p.P = P;
  const long long rows = (long long)batch * T;
  const unsigned grid = (unsigned)(rows < 148 * 8 ? rows : 148 * 8);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  SL_DISPATCH_DTYPE(io_dtype, Tt, {
    if (tail_vec_ok<Tt>(p)) {
      const int pieces = heads * P / Vec16<Tt>::N, threads = (pieces + 31) / 32 * 32;
      if (pieces <= TAIL_THREADS) {   // one piece per thread, just the warps a row fills
        const long long fit = 148ll * (8 * TAIL_THREADS / threads);
        tail_fwd_vec_kernel<Tt, 1><<<(unsigned)(rows < fit ? rows : fit), threads, 0, st>>>(p);
      }
      else tail_fwd_vec_kernel<Tt, 2><<<grid, TAIL_THREADS, 0, st>>>(p);
    } else tail_fwd_kernel<Tt><<<grid, TAIL_THREADS, 0, st>>>(p);
  });
  note_launches(1);
  return launch_status();
}

namespace sl {
int mixer_tail_bwd(const void* Y, const void* gate, int64_t gate_stride, const void* skip, const float* d_skip,
                   const void* norm_weight, float eps, const void* d_normed, void* dY, void* d_gate, int64_t d_gate_stride,
                   void* d_skip_input, float* d_d_skip, float* d_norm_weight, int batch, int heads, int T, int P, int io_dtype,
                   cudaStream_t st) {
  if (int e = tail_check(Y, gate, skip, d_skip, norm_weight, batch, heads, T, P, io_dtype)) return e;
  if (!d_normed || !dY || !d_gate || !d_norm_weight) return SL_ERR_NULL_POINTER;
  TailParams p{};
  p.Y = Y; p.gate = gate; p.skip = skip; p.w = norm_weight; p.d_skip = d_skip; p.dn = d_normed;
  p.dY = dY; p.dgate = d_gate; p.dskip_in = d_skip_input; p.d_d_skip = d_d_skip;
  p.d_w = d_norm_weight; p.gs = gate_stride; p.dgs = d_gate_stride; p.eps = eps;
  p.batch = batch; p.H = heads; p.T = T; p.P = P;
  const long long rows = (long long)batch * T;
  const unsigned grid = (unsigned)(rows < 148 * 2 ? rows : 148 * 2);   // two resident CTAs per SM
  const size_t smem = (size_t)heads * sizeof(float);
  SL_DISPATCH_DTYPE(io_dtype, Tt, {
    const int pieces = heads * P / Vec16<Tt>::N;
    if (tail_vec_ok<Tt>(p)) {
      // one piece per thread; 24 warps per SM stay resident.  16384 rows of 2048 channels: 153 us with an atomic per thread
      // for the sums over rows, 130 with one per head and four weights
      if (pieces <= TAIL_THREADS) {
        const int threads = (pieces + 31) / 32 * 32;
        const long long fit = 148ll * (24 * 32 / threads);
        tail_bwd_row_kernel<Tt><<<(unsigned)(rows < fit ? rows : fit), threads, 0, st>>>(p);
      } else tail_bwd_vec_kernel<Tt, 2><<<grid, TAIL_THREADS, 0, st>>>(p);
    } else tail_bwd_kernel<Tt><<<grid, TAIL_THREADS, smem, st>>>(p);
  });
  note_launches(1);
  return launch_status();
}
}  // namespace sl

extern "C" int sl_mixer_tail_bwd(const void* Y, const void* gate, int64_t gate_row_stride,
                                 const void* skip, const float* d_skip, const void* norm_weight,
                                 float eps, const void* d_normed, void* dY, void* d_gate,
                                 void* d_skip_input, float* d_d_skip, float* d_norm_weight,
                                 int batch, int heads, int T, int P, int io_dtype, void* stream) {
  return sl::mixer_tail_bwd(Y, gate, gate_row_stride, skip, d_skip, norm_weight, eps, d_normed, dY, d_gate,
                            (int64_t)heads * P, d_skip_input, d_d_skip, d_norm_weight, batch, heads, T, P, io_dtype,
                            reinterpret_cast<cudaStream_t>(stream));
}
