// The linear layers of a block's decode token: y = act(x W^T + bias) or residual + x W^T + bias, M <= 64 rows of 16-bit values.
//
// An output has one float32 accumulator, and k ascends in the steps of mma.sync m16n8k16: the plain order, the same for every
// number of rows and every width, so a token does not depend on the batch that it comes in.  (A lane reads 8 consecutive bytes
// of a row for its four values of a step: within a step the order of k is the instruction's own.)  Rounding points are those of
// the composed path: the product is rounded to its type before residual, activation or norm.  The tests hold a block's token to
// the composed path's bits, because a last bit moved here grows from block to block (1.6 % after one token of six blocks of
// width 1024).  A tile is 8 columns, so widths that are no multiple of 8 are left to the library.
//
// What bounds it: the launch.  A library product costs the host 7 to 9 us and a launch of its own for each part of in_proj, the
// residual, the activation and the norm; here it is 2 to 3 us with all of them inside (norms: up to 16 rows).  On the device:
// latency of one trip to memory (all of a warp's rows of W are requested at the start, x two pieces ahead) and the chain of
// K / 16 steps on one accumulator.
#include <algorithm>

#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

// rounded as torch's sums round (no saturation)
template <typename T> __device__ __forceinline__ float rounded(float v);
template <> __device__ __forceinline__ float rounded<__nv_bfloat16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <> __device__ __forceinline__ float rounded<__half>(float v) { return __half2float(__float2half_rn(v)); }
template <typename T> __device__ __forceinline__ uint32_t plain_pair(float a, float b);
template <> __device__ __forceinline__ uint32_t plain_pair<__nv_bfloat16>(float a, float b) { return pack_pair<__nv_bfloat16>(a, b); }
template <> __device__ __forceinline__ uint32_t plain_pair<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int KC = 256;                       // k values of a piece of x
constexpr int X_PITCH = 2 * KC + 32;          // rows 32 bytes off a multiple of 128: 8-byte reads of 4 rows x 32 bytes hit all banks
__host__ __device__ constexpr int w_pitch(int K) { return (2 * K + 127) / 128 * 128 + 32; }

// The norm of the rows of x in shared memory, in place, a warp per row: the additions of rmsnorm_fwd_kernel (partials null) or of
// step_norm_kernel in their order.  Every CTA does it for itself, with more warps than it has
// rows of W for: at 16 rows at most that is shorter than a launch (with the 1 or 2 warps of the product it was longer).
template <typename T>
__device__ __forceinline__ void norm_rows(const TokenLinearArgs& p, uint8_t* s_x, int pitch) {
  const int lane = threadIdx.x & 31, pieces = p.K / 8;
  for (int m = threadIdx.x >> 5; m < p.M; m += blockDim.x >> 5) {
    uint4* row = reinterpret_cast<uint4*>(s_x + m * pitch);
    float ss = 0.f;
    if (p.partials) {
      const float* part = p.partials + (size_t)m * p.n_partials;
      for (int v = 0; v < 8; ++v) {
        float s = 0.f;
        for (int k = 32 * v + lane; k < p.n_partials; k += 256) s += part[k];
        ss += warp_sum(s);
      }
    } else {
      for (int c = lane; c < pieces; c += 32) {
        float v[8];
        unpack16<T>(row[c], v);
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
      }
      ss = warp_sum(ss);
    }
    const float rstd = rsqrtf(ss / (float)p.K + p.norm_eps);
    for (int c = lane; c < pieces; c += 32) {
      float v[8], wv[8];
      unpack16<T>(row[c], v);
      load16<T>(reinterpret_cast<const T*>(p.norm_weight) + 8 * c, wv);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = v[k] * rstd * wv[k];
      store16<T>(reinterpret_cast<T*>(row + c), v);
    }
  }
}

// MT: 16-row tiles of x; NT: 8-row tiles of W per warp (2: value and gate of SwiGLU); NORM: x whole in shared memory
template <typename T, int MT, int NT, bool NORM>
__global__ void __launch_bounds__(NORM ? 256 : 128) token_linear_kernel(TokenLinearArgs p, int nw) {   // nw: warps with rows of W
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  const int K = p.K, wp = w_pitch(K), half = p.O / NT;
  const int o0 = w < nw ? 8 * (blockIdx.x * nw + w) : half;   // this warp's rows of W: o0 .. (+ half)
  uint8_t* const s_x = smem;                                    // [2][16 MT][X_PITCH]
  uint8_t* const s_w = smem + (NORM ? 16 * wp : 2 * 16 * MT * X_PITCH) + (size_t)w * NT * 8 * wp;
  const T* W = reinterpret_cast<const T*>(p.weight);
  grid_release();
  // ---- request this warp's rows of W; k beyond K reads as zero up to the next step ---------------------------------
  const int pieces = (K + 15) / 16 * 2;   // 16-byte pieces of a row
  if (o0 < half)
#pragma unroll 1
    for (int r = 0; r < 8 * NT; ++r) {
      const T* row = W + (size_t)((r >> 3) * half + o0 + (r & 7)) * K;
      for (int c = lane; c < pieces; c += 32) cp_async16(s_w + r * wp + 16 * c, row + (8 * c < K ? 8 * c : 0), 8 * c < K ? 16 : 0);
    }
  cp_async_commit();
  grid_wait();
  // ---- x, two pieces of k ahead ------------------------------------------------------------------------------------
  const int M = p.M, chunks = (K + KC - 1) / KC;
  const T* X = reinterpret_cast<const T*>(p.x);
  auto stage = [&](int c) {
    if (c < chunks)
      for (int i = tid; i < M * (KC / 8); i += blockDim.x) {
        const int m = i / (KC / 8), k = c * KC + 8 * (i % (KC / 8));
        cp_async16(s_x + ((c & 1) * 16 * MT + m) * X_PITCH + 16 * (i % (KC / 8)), X + (size_t)m * K + (k < K ? k : 0), k < K ? 16 : 0);
      }
    cp_async_commit();
  };
  if (NORM) {
    for (int m = 0; m < M; ++m)
      for (int c = tid; c < pieces; c += blockDim.x) cp_async16(s_x + m * wp + 16 * c, X + (size_t)m * K + (8 * c < K ? 8 * c : 0), 8 * c < K ? 16 : 0);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    norm_rows<T>(p, s_x, wp);
    __syncthreads();
  } else {
    stage(0);
    stage(1);
  }
  const int x_pitch = NORM ? wp : X_PITCH, turns = NORM ? 1 : chunks;
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  for (int c = 0; c < turns; ++c) {
    if (!NORM) {
      cp_async_wait<1>();
      __syncthreads();
    }
    if (o0 < half) {
      const uint8_t* xs = s_x + (c & 1) * 16 * MT * X_PITCH + 8 * t;
      const uint8_t* ws = s_w + 2 * c * KC + 8 * t;
      const int steps = ((NORM ? K : min(KC, K - c * KC)) + 15) / 16;
#pragma unroll 4
      for (int s = 0; s < steps; ++s) {
        uint2 b[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) b[j] = *reinterpret_cast<const uint2*>(ws + (8 * j + g) * wp + 32 * s);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const uint2 lo = *reinterpret_cast<const uint2*>(xs + (16 * i + g) * x_pitch + 32 * s);
          const uint2 hi = *reinterpret_cast<const uint2*>(xs + (16 * i + 8 + g) * x_pitch + 32 * s);
          const uint32_t a[4] = {lo.x, hi.x, lo.y, hi.y};   // (rows beyond M hold anything: they reach their own results only)
#pragma unroll
          for (int j = 0; j < NT; ++j) mma16816<T>(acc[i][j], a, b[j].x, b[j].y);
        }
      }
    }
    if (!NORM) {
      __syncthreads();
      stage(c + 2);
    }
  }
  if (o0 >= half) return;
  // ---- epilogue: rounded as the product, then what follows it --------------------------------------------------------
  T* out = reinterpret_cast<T*>(p.out[0]);
  int width = p.width[0], col = o0;
  if (NT == 1) {
    if (col >= width) { col -= width; out = reinterpret_cast<T*>(p.out[1]); width = p.width[1]; }
    if (col >= width && p.out[2]) { col -= width; out = reinterpret_cast<T*>(p.out[2]); width = p.width[2]; }
  }
  const T* bias = reinterpret_cast<const T*>(p.bias);
  float bv[NT][2];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) bv[j][e] = bias ? to_f32(bias[j * half + o0 + 2 * t + e]) : 0.f;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int m = 16 * i + 8 * hh + g;
      if (m >= M) continue;
      float v[NT][2];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          v[j][e] = acc[i][j][2 * hh + e];
          if (bias) v[j][e] += bv[j][e];
        }
      const size_t at = (size_t)m * width + col + 2 * t;
      uint32_t word;
      if (NT == 2) {
        word = pack_pair<T>(rounded<T>(v[0][0]) * silu_f(rounded<T>(v[NT - 1][0])), rounded<T>(v[0][1]) * silu_f(rounded<T>(v[NT - 1][1])));
      } else if (p.gelu) {
        word = pack_pair<T>(gelu_tanh_f<true>(rounded<T>(v[0][0])), gelu_tanh_f<true>(rounded<T>(v[0][1])));
      } else if (p.residual) {
        const float2 r = unpack_pair<T>(*reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(p.residual) + at));
        word = plain_pair<T>(r.x + rounded<T>(v[0][0]), r.y + rounded<T>(v[0][1]));
      } else {
        word = plain_pair<T>(v[0][0], v[0][1]);
      }
      *reinterpret_cast<uint32_t*>(out + at) = word;
    }
}

// Warps with rows of W (8 a warp) of a CTA: one while they still spread over the SMs, more when there are several for each, or
// (without a norm) where that saves a round of CTAs: 64 x 2048 by 4096 columns 29.6 us with two, 15.9 with four.
struct Plan {
  int nw, rounds;   // nw 0: does not fit
  size_t smem;
};
Plan plan_of(const TokenLinearArgs& a) {
  const int NT = a.swiglu ? 2 : 1, MT = (a.M + 15) / 16, tiles = a.O / NT / 8;
  auto bytes = [&](int nw) {
    return (a.norm_weight ? 16 * w_pitch(a.K) : 2 * 16 * (size_t)MT * X_PITCH) + (size_t)nw * NT * 8 * w_pitch(a.K);
  };
  auto rounds = [&](int nw) {   // (four CTAs on an SM at most: more would share its issue slots)
    const int slots = 148 * std::max(1, std::min(4, (int)(227 * 1024 / (bytes(nw) + 1024))));
    return ((tiles + nw - 1) / nw + slots - 1) / slots;
  };
  int nw = tiles <= 2 * 148 ? 1 : tiles <= 8 * 148 ? 2 : 4;
  while (!a.norm_weight && nw < 4 && rounds(2 * nw) < rounds(nw)) nw *= 2;
  while (nw > 0 && bytes(nw) > 200 * 1024) nw /= 2;
  return nw ? Plan{nw, rounds(nw), bytes(nw)} : Plan{0, 0, 0};
}

template <typename T, int MT, int NT, bool NORM>
int launch_token_as(const TokenLinearArgs& a, const Plan& p, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};
  if (int e = ensure_smem(token_linear_kernel<T, MT, NT, NORM>, 200 * 1024, done)) return e;
  const int tiles = a.O / NT / 8;
  // (warps without rows of W help to stage x: 23 x 3840 by 960 columns was bound by one warp's copies)
  return launch_chained(token_linear_kernel<T, MT, NT, NORM>, dim3((tiles + p.nw - 1) / p.nw), NORM ? 256u : 128u, p.smem, st, a.dependent, a, p.nw);
}
template <typename T, int MT>
int launch_token_m(const TokenLinearArgs& a, const Plan& p, cudaStream_t st) {
  if constexpr (MT == 1)
    if (a.norm_weight) return a.swiglu ? launch_token_as<T, 1, 2, true>(a, p, st) : launch_token_as<T, 1, 1, true>(a, p, st);
  return a.swiglu ? launch_token_as<T, MT, 2, false>(a, p, st) : launch_token_as<T, MT, 1, false>(a, p, st);
}
template <typename T>
int launch_token(const TokenLinearArgs& a, const Plan& p, cudaStream_t st) {
  switch ((a.M + 15) / 16) {
    case 1: return launch_token_m<T, 1>(a, p, st);
    case 2: return launch_token_m<T, 2>(a, p, st);
    case 3: return launch_token_m<T, 3>(a, p, st);
    default: return launch_token_m<T, 4>(a, p, st);
  }
}

}  // namespace

// Whole tiles of 8 columns, rows of W that start on 16 bytes, and a chain that is not too long: a warp takes 1.3 us and 1.7 ns for
// each k of each of its 16 x 8 tiles, and CTAs that do not fit on the chip at once take turns.  The library's product is 4 to 10 us on
// the device, and 5 to 7 of host with what follows it as launches of their own.  Device times, here / library: 32 x 1024 by 4096
// columns 7.0 / 6.2, by 16384 16.0 / 10.3; 32 x 4096 by 1024 18.6 / 10.3; 64 x 1024 by 2048 8.8 / 6.2, 64 x 2048 by 2048 16.0 / 8.0.
// So 4096 such k where the norm is inside or the library would need more than a product (in_proj's three parts, the product in
// front of a SwiGLU), 3072 up to 32 rows, 2048 beyond.  Two blocks, us, before this kernel / with one limit of 2048 / of 4096 / none: 24 rows of
// width 960 (gelu, N 128) 216 / 207 / 229 / 228, 48 of 960 (swiglu, N 64) 202 / 201 / 221 / 255, 48 of 768 (swiglu, one group)
// 199 / 187 / 145 / 172, 17 of 768 195 / 135 / 111 / 111, 1 of 1024 196 / 127 / 108 / 108.
bool token_linear_supported(const TokenLinearArgs& a) {
  if (a.M < 1 || a.M > 64 || a.K < 8 || a.K % 8 || a.O < 8 || a.O % (a.swiglu ? 16 : 8) || (a.io_dtype != SL_BF16 && a.io_dtype != SL_F16))
    return false;
  for (int i = 0; i < 3; ++i)
    if (a.width[i] % 8 || !aligned(a.out[i], 4)) return false;
  if (a.norm_weight && (a.M > 16 || !aligned(a.norm_weight, 16) || (!a.partials && a.K > 2048))) return false;
  if (!aligned(a.x, 16) || !aligned(a.weight, 16) || !aligned(a.residual, 4)) return false;
  const Plan p = plan_of(a);
  const int limit = a.M <= 16 || a.out[2] || a.swiglu ? 4096 : a.M <= 32 ? 3072 : 2048;
  return p.nw > 0 && (long long)p.rounds * a.K * ((a.M + 15) / 16) * (a.swiglu ? 2 : 1) <= limit;
}

int token_linear(const TokenLinearArgs& a, cudaStream_t st) {
  if (!a.x || !a.weight || !a.out[0]) return SL_ERR_NULL_POINTER;
  if (!token_linear_supported(a)) return SL_ERR_UNSUPPORTED;
  const Plan p = plan_of(a);
  const int rc = a.io_dtype == SL_BF16 ? launch_token<__nv_bfloat16>(a, p, st) : launch_token<__half>(a, p, st);
  if (rc != SL_OK) return rc;
  note_launches(1);
  return launch_status();
}

}  // namespace sl
