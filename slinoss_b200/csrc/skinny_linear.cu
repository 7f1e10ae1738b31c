// Linear layers of a mixer's decode token: y (M, O) = norm(x) W^T + bias for M <= 64 rows of 16-bit values.
//
// Bound by reading W once (O K 2 bytes); at these sizes also by launches, so the row norm in front of the output projection
// is applied as x is read (its sums of squares come with x).  A library GEMM took 4 to 6 us.
//
// A CTA owns 8 NT output rows; its warps split K in runs of 256.  W is the (n = 8) operand of mma.sync m16n8k16: a
// lane reads 16 consecutive bytes of one row of W (four lanes cover 64 bytes) and uses them for two k-steps under a
// permutation of k that the x fragments share.  All loads of a run are requested before anything else is done, so a
// warp has 4 KB NT in flight; x comes through L1, where all CTAs of an SM find it.  The warps' partial products meet
// in shared memory.  mma.sync, not tcgen05: the tensor pipe idles either way and fragments stay in registers.
#include "common.cuh"
#include "host_abi.h"

namespace sl {
namespace {

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
// MT: 16-row tiles of x; NT: 8-row tiles of W per warp.
// KEEP (with the norm, up to 8 warps): the warp's fragments of x are requested ahead of the row scales that they wait for.
template <typename T, int MT, int NT, bool KEEP>
__global__ void __launch_bounds__(KEEP ? 256 : 512) skinny_linear_kernel(SkinnyArgs p) {
  constexpr int STEPS = KRUN / 32;
  extern __shared__ __align__(16) float s_acc[];      // [warps][16 MT][8 NT]
  __shared__ float s_rstd[16 * MT];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3, o0 = blockIdx.x * 8 * NT;
  const T* W = reinterpret_cast<const T*>(p.weight);

  grid_release();
  // ---- request this warp's run of W ---------------------------------------------------------------------------
  uint4 wv[NT][STEPS];
  const int k0 = w * KRUN + 8 * t;
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int r = o0 + 8 * j + g;
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      wv[j][s] = make_uint4(0u, 0u, 0u, 0u);
      if (r < p.O && k0 + 32 * s < p.K) wv[j][s] = __ldg(reinterpret_cast<const uint4*>(W + (size_t)r * p.K + k0 + 32 * s));
    }
  }
  grid_wait();
  // this CTA's rows
  const int mb = blockIdx.y * 16 * MT, M = min(p.M - mb, 16 * MT);
  const T* X = reinterpret_cast<const T*>(p.x) + (size_t)mb * p.x_stride;
  const T* bias = reinterpret_cast<const T*>(p.bias);
  const bool norm = p.norm_weight != nullptr;
  // the bias of this thread's first output is requested ahead of the product
  const int c0 = tid % (8 * NT);
  const float bias0 = bias && tid < M * 8 * NT && o0 + c0 < p.O ? to_f32(bias[o0 + c0]) : 0.f;
  uint4 xk[KEEP ? STEPS : 1][KEEP ? MT : 1][2];
  if constexpr (KEEP) {
#pragma unroll
    for (int s = 0; s < STEPS; ++s)
#pragma unroll
      for (int i = 0; i < 2 * MT; ++i) {
        xk[s][i / 2][i % 2] = make_uint4(0u, 0u, 0u, 0u);
        if (8 * i + g < M && k0 + 32 * s < p.K)
          xk[s][i / 2][i % 2] = *reinterpret_cast<const uint4*>(X + (size_t)(8 * i + g) * p.x_stride + k0 + 32 * s);
      }
  }
  // ---- row scales of the norm, while W is on its way ------------------------------------------------------------
  if (norm) {
    for (int m = w; m < M; m += nw) {
      float ss = 0.f;
      for (int k = lane; k < p.n_partials; k += 32) ss += p.partials[(size_t)(mb + m) * p.n_partials + k];
      ss = warp_sum(ss);
      if (lane == 0) s_rstd[m] = rsqrtf(ss / (float)p.K + p.norm_eps);
    }
    __syncthreads();
  }
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
  for (int i = 0; i < 2 * MT; ++i) rs[i] = norm && g + 8 * i < M ? s_rstd[g + 8 * i] : 0.f;
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
  for (int idx = tid; idx < M * PITCH; idx += blockDim.x) {
    const int m = idx / PITCH, c = idx % PITCH, o = o0 + c;
    if (o >= p.O) continue;
    float v = 0.f;
    for (int q = 0; q < nw; ++q) v += s_acc[((size_t)q * 16 * MT + m) * PITCH + c];
    if (bias) v += idx == tid ? bias0 : to_f32(bias[o]);
    reinterpret_cast<T*>(p.out)[(size_t)(mb + m) * p.O + o] = from_f32<T>(v);
  }
}

template <typename T, int MT, int NT, bool KEEP>
int launch_skinny_as(const SkinnyArgs& a, cudaStream_t st) {
  const int warps = (a.K + KRUN - 1) / KRUN;
  const size_t smem = (size_t)warps * 16 * MT * 8 * NT * sizeof(float);   // at most 16 warps x 32 rows x 16 columns: 32 KB
  return launch_chained(skinny_linear_kernel<T, MT, NT, KEEP>, dim3((a.O + 8 * NT - 1) / (8 * NT), (a.M + 16 * MT - 1) / (16 * MT)),
                        (unsigned)(32 * warps), smem, st, a.dependent, a);
}
template <typename T, int MT, int NT>
int launch_skinny(const SkinnyArgs& a, cudaStream_t st) {
  if (a.norm_weight && a.K <= 8 * KRUN) return launch_skinny_as<T, MT, NT, true>(a, st);
  return launch_skinny_as<T, MT, NT, false>(a, st);
}
template <typename T>
int launch_skinny_m(const SkinnyArgs& a, cudaStream_t st) {
  // One 16-row tile of x and one 8-row tile of W per warp give the most CTAs and the shortest chain; with 32 and 16 rows a CTA
  // reads half as many bytes per product.  The line lies where the former no longer fit on the chip at once (64 registers per
  // thread, 128 with the norm's fragments kept).  us, small against large tiles: in_proj 512 x 6192 at 48 rows 8.2 / 10.3 and
  // at 64 12.2 / 10.3, 768 x 9288 at 17 rows 12.1 / 10.2, 1024 x 12384 at 64 29.9 / 24.5; out_proj 2048 x 1024 at 32 rows
  // 10.7 / 12.3 and at 33 14.4 / 12.3, 1536 x 768 at 48 12.3 / 14.9 and at 64 19.4 / 15.0, 1024 x 512 at 64 10.3 / 14.3.
  const int warps = (a.K + KRUN - 1) / KRUN, per_sm = (a.norm_weight && warps <= 8 ? 16 : 32) / warps;
  if (a.M <= 16 || (long long)((a.O + 7) / 8) * ((a.M + 15) / 16) <= 148 * per_sm) return launch_skinny<T, 1, 1>(a, st);
  return launch_skinny<T, 2, 2>(a, st);
}

}  // namespace

bool skinny_supported(int M, int K, int O, int io_dtype) {
  return M >= 1 && M <= 64 && K >= 8 && K % 8 == 0 && K <= 16 * KRUN && O >= 1 && (io_dtype == SL_BF16 || io_dtype == SL_F16);
}

int skinny_linear(const SkinnyArgs& a, cudaStream_t st) {
  if (!skinny_supported(a.M, a.K, a.O, a.io_dtype)) return SL_ERR_UNSUPPORTED;
  if (!a.x || !a.weight || !a.out || (a.norm_weight && !a.partials)) return SL_ERR_NULL_POINTER;
  if (!aligned(a.x, 16) || a.x_stride % 8 || !aligned(a.weight, 16) || (a.norm_weight && !aligned(a.norm_weight, 16)))
    return SL_ERR_BAD_ALIGNMENT;
  const int rc = a.io_dtype == SL_BF16 ? launch_skinny_m<__nv_bfloat16>(a, st) : launch_skinny_m<__half>(a, st);
  if (rc != SL_OK) return rc;
  note_launches(1);
  return launch_status();
}

}  // namespace sl
