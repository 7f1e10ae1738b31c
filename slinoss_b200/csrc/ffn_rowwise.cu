// Row-wise kernels of the block's FFN branch: RMSNorm and the activation (GELU-tanh or SwiGLU), forward
// and backward.  With them the FFN branch is rematerialised in the backward pass (only the branch input
// is kept), as the reference does: block_ffn_residual, slinoss/ops/block/training.py:193-354, with the
// kernels of slinoss/ops/block/cute/norm.py:85,173 and activation.py:78,153.  The two GEMMs stay library
// calls in the caller.  All four kernels are HBM-bound: 16-byte accesses, one pass over their rows.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

// a + b, added in float32 and rounded once, without the saturation of from_f32: bit for bit torch's sum of two such tensors
template <typename T>
__device__ __forceinline__ uint4 plain_sum(const uint4& a, const uint4& b) {
  float x[Vec16<T>::N], y[Vec16<T>::N];
  unpack16<T>(a, x); unpack16<T>(b, y);
#pragma unroll
  for (int k = 0; k < Vec16<T>::N; ++k) x[k] += y[k];
  if constexpr (std::is_same<T, __half>::value) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __half2 h = __floats2half2_rn(x[2 * k], x[2 * k + 1]);
      w[k] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    uint4 r;
    store16<T>(reinterpret_cast<T*>(&r), x);
    return r;
  }
}

// out = a + b (a token's residual behind a product that is left to the library): 16 bytes a thread
template <typename T>
__global__ void __launch_bounds__(256) residual_sum_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b,
                                                           uint4* __restrict__ out, long long pieces) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < pieces) out[i] = plain_sum<T>(a[i], b[i]);
}

// out = x * rsqrt(mean(x^2) + eps) * w.  One warp per row; the row stays packed in registers (16-byte
// pieces, MAXP per lane), so it is read once.
template <typename T, int MAXP>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                          T* __restrict__ out, long long rows, int C, float eps) {
  constexpr int V = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int pieces = C / V;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * C);
  uint4 raw[MAXP];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < MAXP; ++i) {
    const int pc = lane + 32 * i;
    if (pc < pieces) raw[i] = xr[pc];
  }
#pragma unroll
  for (int i = 0; i < MAXP; ++i) {
    if (lane + 32 * i < pieces) {
      float v[V];
      unpack16<T>(raw[i], v);
#pragma unroll
      for (int k = 0; k < V; ++k) ss += v[k] * v[k];
    }
  }
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / (float)C + eps);
#pragma unroll
  for (int i = 0; i < MAXP; ++i) {
    const int pc = lane + 32 * i;
    if (pc < pieces) {
      float v[V], wv[V], o[V];
      unpack16<T>(raw[i], v);
      load16<T>(w + pc * V, wv);
#pragma unroll
      for (int k = 0; k < V; ++k) o[k] = v[k] * rstd * wv[k];
      store16<T>(out + row * C + pc * V, o);
    }
  }
}

// dx = rstd (g - xhat mean(g xhat)),  g = dy w,  xhat = x rstd;   dw += sum_rows dy xhat.
// A CTA walks its rows (grid-stride), one warp per row with x and dy packed in registers; every warp adds
// its rows' part of dw into a float row of its own in shared memory (plain 16-byte read-modify-writes: 128
// wavefronts per row against the ~280 cycles the row's bytes take at the SM's share of the HBM bandwidth),
// and the CTA sums the warps' rows and issues one global float atomic per channel at the end.  Keeping dw
// out of the registers leaves room for two CTAs per SM (shared-memory float atomics into one row were
// slower than this, and dw in registers allowed one CTA per SM).  The weight sits packed in shared memory.
template <typename T, int MAXP>
__global__ void __launch_bounds__(256, 2) rmsnorm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                          const T* __restrict__ dy, T* __restrict__ dx,
                                                          float* __restrict__ dw, double* __restrict__ dw64,
                                                          const T* __restrict__ extra, double* __restrict__ extra_sum,
                                                          long long rows, int C, float eps) {
  constexpr int V = Vec16<T>::N;
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* s_dw = reinterpret_cast<float*>(s_raw);                        // [nw][C]
  const int kept = extra_sum ? 2 * nw : nw;                             // rows of sums: dw, then those of extra
  uint4* s_w = reinterpret_cast<uint4*>(s_raw + (size_t)kept * C * sizeof(float));   // [C / V]
  float* my_dw = s_dw + (size_t)warp * C;
  const int pieces = C / V;
  for (int c = threadIdx.x; c < kept * C; c += blockDim.x) s_dw[c] = 0.f;
  for (int c = threadIdx.x; c < pieces; c += blockDim.x) s_w[c] = reinterpret_cast<const uint4*>(w)[c];
  __syncthreads();
  for (long long row = (long long)blockIdx.x * nw + warp; row < rows; row += (long long)gridDim.x * nw) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * C);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + row * C);
    uint4 xraw[MAXP], graw[MAXP];
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      const int pc = lane + 32 * i;
      if (pc < pieces) { xraw[i] = xr[pc]; graw[i] = gr[pc]; }
    }
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      const int pc = lane + 32 * i;
      if (pc < pieces) {
        float xv[V], gv[V], wv[V];
        unpack16<T>(xraw[i], xv); unpack16<T>(graw[i], gv); unpack16<T>(s_w[pc], wv);
#pragma unroll
        for (int k = 0; k < V; ++k) { ss += xv[k] * xv[k]; dot += gv[k] * wv[k] * xv[k]; }
      }
    }
    ss = warp_sum(ss); dot = warp_sum(dot);
    const float rstd = rsqrtf(ss / (float)C + eps);
    const float coef = dot * rstd * rstd / (float)C;     // mean(g xhat) rstd
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      const int pc = lane + 32 * i;
      if (pc < pieces) {
        float xv[V], gv[V], wv[V], o[V];
        unpack16<T>(xraw[i], xv); unpack16<T>(graw[i], gv); unpack16<T>(s_w[pc], wv);
#pragma unroll
        float4* acc = reinterpret_cast<float4*>(my_dw + pc * V);
#pragma unroll
        for (int q = 0; q < V / 4; ++q) {
          float4 a = acc[q];
          a.x += gv[4 * q] * (xv[4 * q] * rstd); a.y += gv[4 * q + 1] * (xv[4 * q + 1] * rstd);
          a.z += gv[4 * q + 2] * (xv[4 * q + 2] * rstd); a.w += gv[4 * q + 3] * (xv[4 * q + 3] * rstd);
          acc[q] = a;
        }
#pragma unroll
        for (int k = 0; k < V; ++k) o[k] = rstd * (gv[k] * wv[k] - xv[k] * coef);
        if (extra) {
          float ev[V];
          load16<T>(extra + row * C + pc * V, ev);
#pragma unroll
          for (int k = 0; k < V; ++k) o[k] += ev[k];
          if (extra_sum) {
            float* es = my_dw + (size_t)nw * C + pc * V;
#pragma unroll
            for (int k = 0; k < V; ++k) es[k] += ev[k];
          }
        }
        store16<T>(dx + row * C + pc * V, o);
      }
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float v = 0.f;
    for (int q = 0; q < nw; ++q) v += s_dw[(size_t)q * C + c];
    if (dw64) atomicAdd(dw64 + c, (double)v);   // the order of these adds is lost in the rounding to the result's type
    else atomicAdd(dw + c, v);
    if (extra_sum) {
      v = 0.f;
      for (int q = nw; q < 2 * nw; ++q) v += s_dw[(size_t)q * C + c];
      atomicAdd(extra_sum + c, (double)v);
    }
  }
}

// Column sums of a (rows, C) matrix, in an order that does not depend on the schedule: each CTA sums a run of rows of 32 V
// columns (a warp per row, 16 bytes a lane) to a row of float32 partials, the second kernel sums those.
template <typename T>
__global__ void __launch_bounds__(256) column_partials_kernel(const T* __restrict__ x, float* __restrict__ partial, long long rows,
                                                              int C, int run) {
  constexpr int V = Vec16<T>::N;
  __shared__ float s_sum[8][32 * V + 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = blockIdx.x * 32 * V, c = c0 + lane * V;
  const long long r0 = (long long)blockIdx.y * run, r1 = min(rows, r0 + run);
  float acc[V];
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = 0.f;
  if (c < C) {
#pragma unroll 4
    for (long long r = r0 + warp; r < r1; r += 8) {
      float v[V];
      load16<T>(x + r * C + c, v);
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += v[k];
    }
  }
#pragma unroll
  for (int k = 0; k < V; ++k) s_sum[warp][lane * V + k] = acc[k];
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * V && c0 + i < C; i += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) v += s_sum[q][i];
    partial[(size_t)blockIdx.y * C + c0 + i] = v;
  }
}
// out[c] = sum of n partial rows: 32 columns per CTA, 8 warps share the rows
template <typename T>
__global__ void __launch_bounds__(256) sum_partials_kernel(const float* __restrict__ partial, T* __restrict__ out, int n, int C) {
  __shared__ float s_sum[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float v = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int r = warp; r < n; r += 8) v += partial[(size_t)r * C + c];
  }
  s_sum[warp][lane] = v;
  __syncthreads();
  if (warp == 0 && c < C) {
    v = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) v += s_sum[q][lane];
    out[c] = from_f32<T>(v);
  }
}

template <bool FAST> __device__ __forceinline__ float dgelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  const float t = tanh_io<FAST>(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
}

// The backward of rows of up to 3 pieces per lane (768 channels of 16-bit rows, 384 of float32): the weight, its gradient and the
// sums of extra stay in registers.  In shared memory (rmsnorm_bwd_kernel) the sums cost a 32-byte read and write per piece and
// row.  What is left is one row's latency per turn and the atomics.  us, bf16, in turn with the kernels of 2 and of 8 pieces that
// these widths had, without / with extra and its sums: 256 rows x 128 4.2 -> 4.2 / 4.4 -> 4.3, 4096 x 256 12.4 -> 6.3 / 14.5 -> 6.4,
// 8192 x 512 16.5 -> 8.4 / 22.8 -> 10.2, 8192 x 576 13.4 -> 10.5 / 22.8 -> 14.7, 16384 x 768 20.8 -> 14.9 / 43.5 -> 26.7; no
// width from 128 to 768 at 256 to 16384 rows got slower, in any type.  With three pieces and the sums 200 bytes are spilled.
template <typename T, int MAXP, bool SUM>
__global__ void __launch_bounds__(512, 1) rmsnorm_bwd_narrow_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                                 const T* __restrict__ dy, T* __restrict__ dx, float* __restrict__ dw,
                                                                 double* __restrict__ dw64, const T* __restrict__ extra,
                                                                 double* __restrict__ extra_sum, long long rows, int C, float eps) {
  constexpr int V = Vec16<T>::N;
  extern __shared__ __align__(16) unsigned char s_raw[];
  float* const s_sum = reinterpret_cast<float*>(s_raw);   // [warps][C]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, pieces = C / V;
  uint4 wr[MAXP];
  f2 sw[MAXP][V / 2], se[SUM ? MAXP : 1][V / 2];
#pragma unroll
  for (int i = 0; i < MAXP; ++i) {
    wr[i] = make_uint4(0u, 0u, 0u, 0u);
    if (lane + 32 * i < pieces) wr[i] = reinterpret_cast<const uint4*>(w)[lane + 32 * i];
#pragma unroll
    for (int k = 0; k < V / 2; ++k) { sw[i][k] = 0ull; if (SUM) se[i][k] = 0ull; }
  }
  for (long long row = (long long)blockIdx.x * nw + warp; row < rows; row += (long long)gridDim.x * nw) {
    uint4 xc[MAXP], gc[MAXP], ec[MAXP];
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      const int pc = lane + 32 * i;
      xc[i] = gc[i] = ec[i] = make_uint4(0u, 0u, 0u, 0u);
      if (pc >= pieces) continue;
      xc[i] = reinterpret_cast<const uint4*>(x + row * C)[pc];
      gc[i] = reinterpret_cast<const uint4*>(dy + row * C)[pc];
      if (extra) ec[i] = reinterpret_cast<const uint4*>(extra + row * C)[pc];
    }
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      float xv[V], gv[V], wv[V];
      unpack16<T>(xc[i], xv); unpack16<T>(gc[i], gv); unpack16<T>(wr[i], wv);
#pragma unroll
      for (int k = 0; k < V; ++k) { ss += xv[k] * xv[k]; dot += gv[k] * wv[k] * xv[k]; }
    }
    ss = warp_sum(ss); dot = warp_sum(dot);
    const float rstd = rsqrtf(ss / (float)C + eps);
    const float coef = dot * rstd * rstd / (float)C;     // mean(g xhat) rstd
    const f2 r2 = dup2(rstd), c2 = dup2(-coef);
#pragma unroll
    for (int i = 0; i < MAXP; ++i) {
      float xv[V], gv[V], wv[V], ev[V], o[V];
      unpack16<T>(xc[i], xv); unpack16<T>(gc[i], gv); unpack16<T>(wr[i], wv);
      if (extra) unpack16<T>(ec[i], ev);
#pragma unroll
      for (int k = 0; k < V / 2; ++k) {
        const f2 x2 = mk2(xv[2 * k], xv[2 * k + 1]), g2 = mk2(gv[2 * k], gv[2 * k + 1]), w2 = mk2(wv[2 * k], wv[2 * k + 1]);
        sw[i][k] = fma2(g2, mul2(x2, r2), sw[i][k]);
        f2 d = mul2(r2, fma2(x2, c2, mul2(g2, w2)));
        if (extra) {
          const f2 e2 = mk2(ev[2 * k], ev[2 * k + 1]);
          d = add2(d, e2);
          if (SUM) se[i][k] = add2(se[i][k], e2);
        }
        const float2 q = un2(d);
        o[2 * k] = q.x; o[2 * k + 1] = q.y;
      }
      if (lane + 32 * i < pieces) store16<T>(dx + row * C + (lane + 32 * i) * V, o);
    }
  }
#pragma unroll
  for (int part = 0; part < (SUM ? 2 : 1); ++part) {
#pragma unroll
    for (int i = 0; i < MAXP; ++i)
      if (lane + 32 * i < pieces)
#pragma unroll
        for (int k = 0; k < V / 2; ++k)
          *reinterpret_cast<f2*>(s_sum + (size_t)warp * C + (lane + 32 * i) * V + 2 * k) = part ? se[SUM ? i : 0][k] : sw[i][k];
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      double v = 0.0;
      for (int q = 0; q < nw; ++q) v += s_sum[(size_t)q * C + c];
      if (part) atomicAdd(extra_sum + c, v);
      else if (dw64) atomicAdd(dw64 + c, v);   // the order of these adds is lost in the rounding to the result's type
      else atomicAdd(dw + c, (float)v);
    }
    __syncthreads();
  }
}

// kind 0: hidden = gelu_tanh(projected) (same width).  kind 1 (SwiGLU): projected = [value | gate] of
// width 2 H per row, hidden = value * silu(gate).  One 16-byte piece of the hidden row per thread.
template <typename T>
__global__ void __launch_bounds__(256) ffn_act_fwd_kernel(const T* __restrict__ proj, T* __restrict__ hidden,
                                                          long long rows, int H, int kind) {
  constexpr int V = Vec16<T>::N;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int ppr = H / V;
  if (i >= rows * ppr) return;
  const long long row = i / ppr;
  const int pc = (int)(i % ppr);
  float a[V], o[V];
  if (kind == 0) {
    load16<T>(proj + row * H + pc * V, a);
#pragma unroll
    for (int k = 0; k < V; ++k) o[k] = gelu_tanh_f<sizeof(T) == 2>(a[k]);
  } else {
    float g[V];
    load16<T>(proj + row * 2 * H + pc * V, a);
    load16<T>(proj + row * 2 * H + H + pc * V, g);
#pragma unroll
    for (int k = 0; k < V; ++k) o[k] = a[k] * silu_f(g[k]);
  }
  store16<T>(hidden + row * H + pc * V, o);
}

template <typename T>
__global__ void __launch_bounds__(256) ffn_act_bwd_kernel(const T* __restrict__ proj, const T* __restrict__ dhid,
                                                          T* __restrict__ dproj, long long rows, int H, int kind) {
  constexpr int V = Vec16<T>::N;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int ppr = H / V;
  if (i >= rows * ppr) return;
  const long long row = i / ppr;
  const int pc = (int)(i % ppr);
  float a[V], d[V], o[V];
  load16<T>(dhid + row * H + pc * V, d);
  if (kind == 0) {
    load16<T>(proj + row * H + pc * V, a);
#pragma unroll
    for (int k = 0; k < V; ++k) o[k] = d[k] * dgelu_tanh_f<sizeof(T) == 2>(a[k]);
    store16<T>(dproj + row * H + pc * V, o);
  } else {
    float g[V], og[V];
    load16<T>(proj + row * 2 * H + pc * V, a);
    load16<T>(proj + row * 2 * H + H + pc * V, g);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float s = sigmoid_f(g[k]);
      o[k] = d[k] * g[k] * s;                                  // d value
      og[k] = d[k] * a[k] * (s + g[k] * s * (1.f - s));        // d gate
    }
    store16<T>(dproj + row * 2 * H + pc * V, o);
    store16<T>(dproj + row * 2 * H + H + pc * V, og);
  }
}

// The activation's backward with the column sums of its result (the bias gradient of the projection): a CTA walks a run of rows
// of 32 V columns, a warp per row, and adds its float32 sums to float64 accumulators once.  The elementwise kernel above followed by a
// pass for the sums reads the result again (8192 x 2304: 24 + 15 us, now 24).
template <typename T>
__global__ void __launch_bounds__(256) ffn_act_bwd_sum_kernel(const T* __restrict__ proj, const T* __restrict__ dhid,
                                                              T* __restrict__ dproj, double* __restrict__ sums, long long rows,
                                                              int H, int kind, int run) {
  constexpr int V = Vec16<T>::N;
  __shared__ float s_sum[8][32 * V + 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = blockIdx.x * 32 * V, c = c0 + lane * V;
  const long long r0 = (long long)blockIdx.y * run, r1 = min(rows, r0 + run);
  const size_t pitch = (size_t)(kind ? 2 : 1) * H;
  float acc[V], acg[V];
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = acg[k] = 0.f;
  if (c < H) {
#pragma unroll 2
    for (long long r = r0 + warp; r < r1; r += 8) {
      float a[V], d[V], o[V];
      load16<T>(dhid + r * H + c, d);
      load16<T>(proj + r * pitch + c, a);
      if (kind == 0) {
#pragma unroll
        for (int k = 0; k < V; ++k) o[k] = d[k] * dgelu_tanh_f<sizeof(T) == 2>(a[k]);
      } else {
        float g[V], og[V];
        load16<T>(proj + r * pitch + H + c, g);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float sg = sigmoid_f(g[k]);
          o[k] = d[k] * g[k] * sg;
          og[k] = d[k] * a[k] * (sg + g[k] * sg * (1.f - sg));
          acg[k] += og[k];
        }
        store16<T>(dproj + r * pitch + H + c, og);
      }
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += o[k];
      store16<T>(dproj + r * pitch + c, o);
    }
  }
  for (int part = 0; part <= kind; ++part) {
#pragma unroll
    for (int k = 0; k < V; ++k) s_sum[warp][lane * V + k] = part ? acg[k] : acc[k];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * V && c0 + i < H; i += blockDim.x) {
      float v = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) v += s_sum[q][i];
      atomicAdd(sums + (size_t)part * H + c0 + i, (double)v);
    }
    __syncthreads();
  }
}

constexpr int RMS_MAXP_NARROW = 2;   // rows up to 512 (256) channels keep the registers low
constexpr int RMS_MAXP = 8;   // 16-byte pieces per lane: rows up to 8 * 32 * (4 or 8) channels

bool rows_ok(long long rows, int C, int dt, const void* a, const void* b) {
  const int V = dt == SL_F32 ? 4 : 8;
  return rows >= 1 && C >= V && C % V == 0 && C / V <= 32 * RMS_MAXP && aligned(a, 16) && aligned(b, 16);
}

}  // namespace
}  // namespace sl

extern "C" int sl_rmsnorm_fwd(const void* x, const void* weight, float eps, void* out, long long rows, int C,
                              int io_dtype, void* stream) {
  using namespace sl;
  if (!x || !weight || !out) return SL_ERR_NULL_POINTER;
  if (!dtype_ok(io_dtype)) return SL_ERR_UNSUPPORTED;
  if (!rows_ok(rows, C, io_dtype, x, out) || !aligned(weight, 16)) return SL_ERR_BAD_SHAPE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((rows + 7) / 8);
  const bool narrow = C / (io_dtype == SL_F32 ? 4 : 8) <= 32 * RMS_MAXP_NARROW;
  SL_DISPATCH_DTYPE(io_dtype, T, {
    auto kern = narrow ? rmsnorm_fwd_kernel<T, RMS_MAXP_NARROW> : rmsnorm_fwd_kernel<T, RMS_MAXP>;
    kern<<<grid, 256, 0, st>>>(reinterpret_cast<const T*>(x), reinterpret_cast<const T*>(weight),
                               reinterpret_cast<T*>(out), rows, C, eps);
  });
  note_launches(1);
  return launch_status();
}

namespace sl {
int residual_sum(const void* a, const void* b, void* out, long long n, int io_dtype, cudaStream_t st) {
  if (!a || !b || !out) return SL_ERR_NULL_POINTER;
  if (!dtype_ok(io_dtype)) return SL_ERR_UNSUPPORTED;
  const int V = io_dtype == SL_F32 ? 4 : 8;
  if (n < V || n % V || !aligned(a, 16) || !aligned(b, 16) || !aligned(out, 16)) return SL_ERR_BAD_SHAPE;
  const long long pieces = n / V;
  SL_DISPATCH_DTYPE(io_dtype, T, {
    residual_sum_kernel<T><<<(unsigned)((pieces + 255) / 256), 256, 0, st>>>(
        reinterpret_cast<const uint4*>(a), reinterpret_cast<const uint4*>(b), reinterpret_cast<uint4*>(out), pieces);
  });
  note_launches(1);
  return launch_status();
}

// d_weight: float32 accumulators, or float64 ones (weight64); extra (or null) is added to d_x, its column sums to extra_sum
// (or null; up to 1024 columns, where the second row of sums per warp still leaves three CTAs per SM)
bool rmsnorm_bwd_sums_extra(int C) { return C <= 1024; }
int rmsnorm_bwd(const void* x, const void* weight, float eps, const void* d_out, const void* extra, void* d_x, float* d_weight,
                double* weight64, double* extra_sum, long long rows, int C, int io_dtype, cudaStream_t st) {
  if (!x || !weight || !d_out || !d_x || !(d_weight || weight64)) return SL_ERR_NULL_POINTER;
  if (!dtype_ok(io_dtype)) return SL_ERR_UNSUPPORTED;
  if (!rows_ok(rows, C, io_dtype, x, d_x) || !aligned(weight, 16) || !aligned(d_out, 16) || !aligned(extra, 16)) return SL_ERR_BAD_SHAPE;
  const long long want = (rows + 7) / 8;
  const int lanes = (C / (io_dtype == SL_F32 ? 4 : 8) + 31) / 32;   // pieces per lane
  if (extra_sum && (!extra || !rmsnorm_bwd_sums_extra(C))) return SL_ERR_UNSUPPORTED;
  if (lanes <= 3) {
    const unsigned grid = (unsigned)std::min<long long>((rows + 15) / 16, 148);   // 16 warps each: half the atomics of 8
    SL_DISPATCH_DTYPE(io_dtype, T, {
      const T *tx = reinterpret_cast<const T*>(x), *tw = reinterpret_cast<const T*>(weight), *td = reinterpret_cast<const T*>(d_out);
      const T* te = reinterpret_cast<const T*>(extra);
      T* to = reinterpret_cast<T*>(d_x);
      auto kern = extra_sum ? (lanes <= 2 ? rmsnorm_bwd_narrow_kernel<T, 2, true> : rmsnorm_bwd_narrow_kernel<T, 3, true>)
                            : (lanes <= 2 ? rmsnorm_bwd_narrow_kernel<T, 2, false> : rmsnorm_bwd_narrow_kernel<T, 3, false>);
      const size_t smem = (size_t)16 * C * sizeof(float);   // (48 KB at most)
      kern<<<grid, 512, smem, st>>>(tx, tw, td, to, d_weight, weight64, te, extra_sum, rows, C, eps);
    });
    note_launches(1);
    return launch_status();
  }
  const long long cap = 148 * 2;   // CTAs that walk the rows: all resident at once
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  const size_t smem = (size_t)(extra_sum ? 16 : 8) * C * sizeof(float) + (size_t)C * dtype_size(io_dtype);   // 8 warps' rows + w
  SL_DISPATCH_DTYPE(io_dtype, T, {
    auto kern = rmsnorm_bwd_kernel<T, RMS_MAXP>;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return SL_ERR_LAUNCH_FAILED;
    kern<<<grid, 256, smem, st>>>(
        reinterpret_cast<const T*>(x), reinterpret_cast<const T*>(weight), reinterpret_cast<const T*>(d_out),
        reinterpret_cast<T*>(d_x), d_weight, weight64, reinterpret_cast<const T*>(extra), extra_sum, rows, C, eps);
  });
  note_launches(1);
  return launch_status();
}

// runs of rows: 8 at least per warp, and about four CTAs per SM
static int column_runs(long long rows, int C, int io) {
  const int cols = (C + 32 * (io == SL_F32 ? 4 : 8) - 1) / (32 * (io == SL_F32 ? 4 : 8));
  const long long most = (rows + 63) / 64, want = (592 + cols - 1) / cols;
  return (int)(most < want ? most : want);
}
int ffn_act_bwd_sum(const void* projected, const void* d_hidden, void* d_projected, double* sums, long long rows, int H, int kind,
                    int io_dtype, cudaStream_t st) {
  const int V = io_dtype == SL_F32 ? 4 : 8, runs = column_runs(rows, H, io_dtype);
  if (rows < 1 || H < V || H % V || !aligned(projected, 16) || !aligned(d_hidden, 16) || !aligned(d_projected, 16)) return SL_ERR_BAD_SHAPE;
  const int run = (int)((rows + runs - 1) / runs);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    ffn_act_bwd_sum_kernel<T><<<dim3((H + 32 * V - 1) / (32 * V), runs), 256, 0, st>>>(
        reinterpret_cast<const T*>(projected), reinterpret_cast<const T*>(d_hidden), reinterpret_cast<T*>(d_projected), sums, rows, H,
        kind, run);
  });
  note_launches(1);
  return launch_status();
}
size_t column_sum_partials(long long rows, int C, int io_dtype) { return (size_t)column_runs(rows, C, io_dtype) * C; }
int column_sum(const void* x, void* out, float* partial, long long rows, int C, int io_dtype, cudaStream_t st) {
  if (!x || !out || !partial) return SL_ERR_NULL_POINTER;
  const int V = io_dtype == SL_F32 ? 4 : 8, runs = column_runs(rows, C, io_dtype);
  if (rows < 1 || C < 1 || C % V || !aligned(x, 16)) return SL_ERR_BAD_SHAPE;
  const int run = (int)((rows + runs - 1) / runs);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    column_partials_kernel<T><<<dim3((C + 32 * V - 1) / (32 * V), runs), 256, 0, st>>>(reinterpret_cast<const T*>(x), partial, rows, C, run);
  });
  note_launches(1);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    sum_partials_kernel<T><<<(C + 31) / 32, 256, 0, st>>>(partial, reinterpret_cast<T*>(out), runs, C);
  });
  note_launches(1);
  return launch_status();
}
}  // namespace sl

extern "C" int sl_rmsnorm_bwd(const void* x, const void* weight, float eps, const void* d_out, void* d_x,
                              float* d_weight, long long rows, int C, int io_dtype, void* stream) {
  return sl::rmsnorm_bwd(x, weight, eps, d_out, nullptr, d_x, d_weight, nullptr, nullptr, rows, C, io_dtype,
                         reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int sl_ffn_activation_fwd(const void* projected, void* hidden, long long rows, int hidden_dim,
                                     int kind, int io_dtype, void* stream) {
  using namespace sl;
  if (!projected || !hidden) return SL_ERR_NULL_POINTER;
  if (!dtype_ok(io_dtype) || (kind != 0 && kind != 1)) return SL_ERR_UNSUPPORTED;
  const int V = io_dtype == SL_F32 ? 4 : 8;
  if (rows < 1 || hidden_dim < V || hidden_dim % V || !aligned(projected, 16) || !aligned(hidden, 16))
    return SL_ERR_BAD_SHAPE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long n = rows * (hidden_dim / V);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    ffn_act_fwd_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        reinterpret_cast<const T*>(projected), reinterpret_cast<T*>(hidden), rows, hidden_dim, kind);
  });
  note_launches(1);
  return launch_status();
}

extern "C" int sl_ffn_activation_bwd(const void* projected, const void* d_hidden, void* d_projected,
                                     long long rows, int hidden_dim, int kind, int io_dtype, void* stream) {
  using namespace sl;
  if (!projected || !d_hidden || !d_projected) return SL_ERR_NULL_POINTER;
  if (!dtype_ok(io_dtype) || (kind != 0 && kind != 1)) return SL_ERR_UNSUPPORTED;
  const int V = io_dtype == SL_F32 ? 4 : 8;
  if (rows < 1 || hidden_dim < V || hidden_dim % V || !aligned(projected, 16) || !aligned(d_hidden, 16) ||
      !aligned(d_projected, 16))
    return SL_ERR_BAD_SHAPE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long n = rows * (hidden_dim / V);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    ffn_act_bwd_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        reinterpret_cast<const T*>(projected), reinterpret_cast<const T*>(d_hidden),
        reinterpret_cast<T*>(d_projected), rows, hidden_dim, kind);
  });
  note_launches(1);
  return launch_status();
}
