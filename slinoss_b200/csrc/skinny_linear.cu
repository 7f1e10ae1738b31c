// Linear layers of a decode token: y (M, O) = act(norm(x) W^T + bias) (+ residual) for M <= 64 rows of 16-bit values.
//
// Bound by reading W once (O K 2 bytes); at these sizes also by launches, so what surrounds the product - RMSNorm of
// the input, bias, activation, residual - happens inside.  A library GEMM pads M to its tile and took 4 to 6 us for
// each of the five products of a block; the norms, the activation and the residual were launches of their own.
//
// A CTA owns 8 NT output rows; its warps split K in runs of 256.  W is the (n = 8) operand of mma.sync m16n8k16: a
// lane reads 16 consecutive bytes of one row of W (four lanes cover 64 bytes) and uses them for two k-steps under a
// permutation of k that the x fragments share.  All loads of a run are requested before anything else is done, so a
// warp has 4 KB NT in flight; x comes through L1, where all CTAs of an SM find it.  The warps' partial products meet
// in shared memory.  mma.sync, not tcgen05: the tensor pipe idles either way and fragments stay in registers.
#include <atomic>

#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

template <typename T> __device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename T> __device__ __forceinline__ float round_io(float v) { return to_f32(from_f32<T>(v)); }
template <typename T> __device__ __forceinline__ uint4 scale_pieces(uint4 x, float s, uint4 w) {   // round(x s w)
  float xv[8], wv[8];
  unpack16<T>(x, xv);
  unpack16<T>(w, wv);
  uint4 o;
  uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int k = 0; k < 4; ++k) ow[k] = pack_pair<T>(xv[2 * k] * s * wv[2 * k], xv[2 * k + 1] * s * wv[2 * k + 1]);
  return o;
}

constexpr int KRUN = 256;                 // k values of a warp
// MT: 16-row tiles of x; NT: 8-row tiles of W per warp (SwiGLU: NT / 2 of values and as many of gates).
// KEEP (with a norm, up to 8 warps and 32 rows): the warp's fragments of x stay in registers, so that x is read once and its
// sums of squares come from there; a pass of its own over x put a load and a reduction per row and warp in front of the
// product (width 512, 8 rows: 7.1 -> 5.4 us per kernel).
template <typename T, int MT, int NT, bool SWIGLU, bool KEEP>
__global__ void __launch_bounds__(KEEP ? 256 : 512) skinny_linear_kernel(SkinnyArgs p) {
  constexpr int STEPS = KRUN / 32;
  constexpr int OT = SWIGLU ? NT / 2 : NT;            // output tiles of the CTA
  extern __shared__ __align__(16) float s_acc[];      // [warps][16 MT][8 NT]
  __shared__ float s_rstd[64], s_ss[KEEP ? 8 : 1][16 * MT];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3, o0 = blockIdx.x * 8 * OT;
  const T* W = reinterpret_cast<const T*>(p.weight);

  grid_release();
  // ---- request this warp's run of W ---------------------------------------------------------------------------
  uint4 wv[NT][STEPS];
  const int k0 = w * KRUN + 8 * t;
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int r = (SWIGLU && j >= OT ? p.O + o0 + 8 * (j - OT) : o0 + 8 * j) + g;
    const bool row_ok = o0 + 8 * (SWIGLU && j >= OT ? j - OT : j) + g < p.O;
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      wv[j][s] = make_uint4(0u, 0u, 0u, 0u);
      if (row_ok && k0 + 32 * s < p.K) wv[j][s] = __ldg(reinterpret_cast<const uint4*>(W + (size_t)r * p.K + k0 + 32 * s));
    }
  }
  grid_wait();
  // this CTA's rows
  const int mb = blockIdx.y * 16 * MT, M = min(p.M - mb, 16 * MT);
  const T* X = reinterpret_cast<const T*>(p.x) + (size_t)mb * p.x_stride;
  const float* partials = p.partials ? p.partials + (size_t)mb * p.n_partials : nullptr;
  const T *bias = reinterpret_cast<const T*>(p.bias), *residual = reinterpret_cast<const T*>(p.residual);
  if (residual) residual += (size_t)mb * p.O;
  // ---- row scales of the norm, while W is on its way ------------------------------------------------------------
  const bool norm = p.norm_weight != nullptr;
  // the first output of this thread: its residual and bias are requested ahead of the product
  const int m0 = tid / (8 * OT), c0 = tid % (8 * OT);
  const bool out0 = tid < M * 8 * OT && o0 + c0 < p.O;
  const float res0 = out0 && residual ? to_f32(residual[(size_t)m0 * p.O + o0 + c0]) : 0.f;
  const float bias0 = out0 && bias ? to_f32(bias[o0 + c0]) : 0.f;
  uint4 xk[KEEP ? STEPS : 1][KEEP ? MT : 1][2];
  if constexpr (KEEP) {
    float sq[2 * MT];
#pragma unroll
    for (int i = 0; i < 2 * MT; ++i) sq[i] = 0.f;
#pragma unroll
    for (int s = 0; s < STEPS; ++s)
#pragma unroll
      for (int i = 0; i < 2 * MT; ++i) {
        xk[s][i / 2][i % 2] = make_uint4(0u, 0u, 0u, 0u);
        if (8 * i + g < M && k0 + 32 * s < p.K)
          xk[s][i / 2][i % 2] = *reinterpret_cast<const uint4*>(X + (size_t)(8 * i + g) * p.x_stride + k0 + 32 * s);
      }
    if (!partials) {
#pragma unroll
      for (int s = 0; s < STEPS; ++s)
#pragma unroll
        for (int i = 0; i < 2 * MT; ++i) {
          float v[8];
          unpack16<T>(xk[s][i / 2][i % 2], v);
#pragma unroll
          for (int q = 0; q < 8; ++q) sq[i] += v[q] * v[q];
        }
#pragma unroll
      for (int i = 0; i < 2 * MT; ++i) {
        sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 1);
        sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 2);
        if (t == 0) s_ss[w][8 * i + g] = sq[i];
      }
    }
  }
  if (norm && !(KEEP && !partials)) {
    for (int m = w; m < M; m += nw) {
      float ss = 0.f;
      if (partials) {
        for (int k = lane; k < p.n_partials; k += 32) ss += partials[(size_t)m * p.n_partials + k];
      } else {
        for (int k = 8 * lane; k < p.K; k += 256) {
          float v[8];
          load16<T>(X + (size_t)m * p.x_stride + k, v);
#pragma unroll
          for (int q = 0; q < 8; ++q) ss += v[q] * v[q];
        }
      }
      ss = warp_sum(ss);
      if (lane == 0) s_rstd[m] = rsqrtf(ss / (float)p.K + p.norm_eps);
    }
  }
  if (norm) __syncthreads();
  // ---- products ---------------------------------------------------------------------------------------------------
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  float rs[2 * MT];
#pragma unroll
  for (int i = 0; i < 2 * MT; ++i) {
    rs[i] = 0.f;
    if (!norm || g + 8 * i >= M) continue;
    if (KEEP && !partials) {
      float ss = 0.f;
      for (int q = 0; q < nw; ++q) ss += s_ss[q][8 * i + g];
      rs[i] = rsqrtf(ss / (float)p.K + p.norm_eps);
    } else {
      rs[i] = s_rstd[g + 8 * i];
    }
  }
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int k = k0 + 32 * s;
    if (w * KRUN + 32 * s >= p.K) break;
    uint4 nwv = make_uint4(0u, 0u, 0u, 0u);
    if (norm && k < p.K) nwv = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.norm_weight) + k));
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      uint4 xa[2];
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int m = 16 * i + 8 * hh + g;
        xa[hh] = make_uint4(0u, 0u, 0u, 0u);
        if (m < M && k < p.K) {
          if constexpr (KEEP) xa[hh] = xk[s][i][hh];
          else xa[hh] = *reinterpret_cast<const uint4*>(X + (size_t)m * p.x_stride + k);
          if (norm) xa[hh] = scale_pieces<T>(xa[hh], rs[2 * i + hh], nwv);
        }
      }
      const uint32_t a0[4] = {xa[0].x, xa[1].x, xa[0].y, xa[1].y}, a1[4] = {xa[0].z, xa[1].z, xa[0].w, xa[1].w};
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma16816<T>(acc[i][j], a0, wv[j][s].x, wv[j][s].y);
        mma16816<T>(acc[i][j], a1, wv[j][s].z, wv[j][s].w);
      }
    }
  }
  // ---- sum over the warps, epilogue -----------------------------------------------------------------------------
  constexpr int PITCH = 8 * NT;
  float* mine = s_acc + (size_t)w * 16 * MT * PITCH;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
        *reinterpret_cast<float2*>(mine + (16 * i + 8 * hh + g) * PITCH + 8 * j + 2 * t) =
            make_float2(acc[i][j][2 * hh], acc[i][j][2 * hh + 1]);
  __syncthreads();
  for (int idx = tid; idx < M * 8 * OT; idx += blockDim.x) {
    const int m = idx / (8 * OT), c = idx % (8 * OT), o = o0 + c;
    if (o >= p.O) continue;
    float v = 0.f, gate = 0.f;
    for (int q = 0; q < nw; ++q) {
      v += s_acc[((size_t)q * 16 * MT + m) * PITCH + c];
      if (SWIGLU) gate += s_acc[((size_t)q * 16 * MT + m) * PITCH + 8 * OT + c];
    }
    if (bias) { v += idx == tid ? bias0 : to_f32(bias[o]); if (SWIGLU) gate += to_f32(bias[p.O + o]); }
    v = round_io<T>(v);
    if (SWIGLU) v = v * silu_f(round_io<T>(gate));
    else if (p.act == LINEAR_GELU) v = gelu_tanh_f<true>(v);
    if (residual) v = round_io<T>(v) + (idx == tid ? res0 : to_f32(residual[(size_t)m * p.O + o]));
    reinterpret_cast<T*>(p.out)[(size_t)(mb + m) * p.O + o] = from_f32<T>(v);
  }
}

template <typename T, int MT, int NT, bool SWIGLU, bool KEEP>
int launch_skinny_as(const SkinnyArgs& a, cudaStream_t st) {
  auto k = skinny_linear_kernel<T, MT, NT, SWIGLU, KEEP>;
  const int warps = (a.K + KRUN - 1) / KRUN;
  const size_t smem = (size_t)warps * 16 * MT * 8 * NT * sizeof(float);
  static std::atomic<unsigned long long> done{0};
  if (smem > 48 * 1024) {
    if (int e = ensure_smem(k, 16 * 16 * MT * 8 * NT * sizeof(float), done)) return e;
  }
  const int rows = 8 * (SWIGLU ? NT / 2 : NT);
  return launch_chained(k, dim3((a.O + rows - 1) / rows, (a.M + 16 * MT - 1) / (16 * MT)), (unsigned)(32 * warps), smem, st, a.dependent, a);
}
template <typename T, int MT, int NT, bool SWIGLU>
int launch_skinny(const SkinnyArgs& a, cudaStream_t st) {
  if (a.norm_weight && a.K <= 8 * KRUN) return launch_skinny_as<T, MT, NT, SWIGLU, true>(a, st);
  return launch_skinny_as<T, MT, NT, SWIGLU, false>(a, st);
}
template <typename T>
int launch_skinny_m(const SkinnyArgs& a, cudaStream_t st) {
  // One 16-row tile of x and one 8-row tile of W per warp give the most CTAs and the shortest chain.  A CTA then reads 48 K
  // bytes, and with many rows of a large layer that traffic takes longer than the chain (width 1024: 348 against 358 us per token
  // of four blocks at 32 rows, 588 against 523 at 64; width 512: 284 against 346 at 64).
  const bool sw = a.act == LINEAR_SWIGLU;
  if (a.M <= 16 || (long long)a.M * a.K * a.O <= 120000000)
    return sw ? launch_skinny<T, 1, 2, true>(a, st) : launch_skinny<T, 1, 1, false>(a, st);
  return sw ? launch_skinny<T, 2, 2, true>(a, st) : launch_skinny<T, 2, 2, false>(a, st);
}

}  // namespace

bool skinny_supported(int M, int K, int O, int io_dtype) {
  return M >= 1 && M <= 64 && K >= 8 && K % 8 == 0 && K <= 16 * KRUN && O >= 1 && (io_dtype == SL_BF16 || io_dtype == SL_F16);
}

int skinny_linear(const SkinnyArgs& a, cudaStream_t st) {
  if (!skinny_supported(a.M, a.K, a.O, a.io_dtype)) return SL_ERR_UNSUPPORTED;
  if (!a.x || !a.weight || !a.out) return SL_ERR_NULL_POINTER;
  if (!aligned(a.x, 16) || a.x_stride % 8 || !aligned(a.weight, 16) || (a.norm_weight && !aligned(a.norm_weight, 16)))
    return SL_ERR_BAD_ALIGNMENT;
  const int rc = a.io_dtype == SL_BF16 ? launch_skinny_m<__nv_bfloat16>(a, st) : launch_skinny_m<__half>(a, st);
  if (rc != SL_OK) return rc;
  note_launches(1);
  return launch_status();
}

}  // namespace sl
