// One decode token of the whole mixer between in_proj and out_proj, in one launch up to the row norm:
//
//   causal conv update + bias + SiLU  ->  u          (per channel, carried conv window)
//   scan preparation of the token     ->  m, kp, kc  (per head)   and  b, c  (per group)
//   state update + read-out            z' = m z + u_prev (x) (kp b_prev) + u (x) (kc b),  y = Re<c, z'>
//   skip + gate                        hid = (y + d_skip u) SiLU(gate)
//   RMSNorm over the inner width       normed = hid * rsqrt(mean hid^2 + eps) * w
//
// (what run_reference_decode_step evaluates with separate torch ops, slinoss/ops/mixer/step.py:201-258 and
// 323-429, and what mixer_decode_step_cute fuses for d_skip-free mixers only,
// slinoss/ops/v2x2ssd/cute/step.py:224-627; the projections are the caller's.)
//
// The RMSNorm needs the sum of squares over ALL heads of a batch row: the step kernels leave the gated values of the
// row and eight partial sums of squares per head (plain stores, no atomics, so a token is bit-reproducible); whoever
// consumes them adds the partials up - the normalising kernel at the end of this file, or the output projection of
// skinny_linear.cu, which applies the norm as it reads its operand.
//
// Values are rounded to the io dtype where the sequence kernels round them (u, b, c, y, the skip sum, the
// gated value), so that a decoded token equals the same token of a forward pass.
#include <atomic>

#include "common.cuh"
#include "host_abi.h"
#include "tc_common.cuh"

namespace sl {
namespace {

__device__ int g_step_status = 0;

#include "scanprep_math.cuh"

template <typename T> __device__ __forceinline__ float round_io(float v) { return to_f32(from_f32<T>(v)); }

struct StepParams {
  const void *gate, *value;          // (batch, C) with row strides (column slices of the in_proj output)
  long long gate_stride, value_stride;
  const void *params, *bc;           // (batch, 3H), (batch, G, 4, N)
  const void *conv_w, *conv_b;       // (C, W), (C)
  void* conv_state;                  // (batch, C, W-1), updated in place
  const float *dt_bias, *alpha_bias, *theta_mod_bias, *theta_bias, *theta_sign, *d_skip;
  const void* norm_w;                // (C)
  sl_scanprep_config cfg;
  float norm_eps;
  float* state;                      // (batch, H, P, 2N), updated in place
  const void* b_prev_in;             // (batch, G, 2N)
  void* b_prev_out;                  // (batch, G, 2N): this token's b (a buffer of its own: heads of a group race otherwise)
  void* u_prev;                      // (batch, H, P), updated in place
  void* hid;                         // (batch, C): gated values, before the row norm
  float* part;                       // (batch, H, 8): partial sums of squares of hid
  long long params_stride, bc_stride;
  int batch, H, G, P, N, W;
};

template <typename T>
__global__ void __launch_bounds__(256, 4) mixer_step_kernel(StepParams p) {
  extern __shared__ __align__(16) float smem[];
  const int D = 2 * p.N, C = p.H * p.P;
  float* s_bp = smem;            // kp * b_prev
  float* s_bc = smem + D;        // kc * b
  float* s_c = smem + 2 * D;     // c
  float* s_b = smem + 3 * D;     // b (rounded)
  float* s_u = smem + 4 * D;     // [P] u, then [P] u_prev, then [P] y
  float* s_up = s_u + p.P;
  float* s_y = s_up + p.P;
  __shared__ float s_coef[6];    // m, kp, kc
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const int g = h / (p.H / p.G);
  const size_t bg = (size_t)b * p.G + g;

  // ---- requests.  Nothing below depends on anything but the inputs until phase D, so every global value
  // the phases A, C, D, E and F read is requested here, ahead of any arithmetic: the CTA then pays for one
  // round trip to memory instead of one per phase (the phases are separated by barriers, and a CTA per
  // (batch, head) has too little work to hide five of them).
  float* state = p.state + (size_t)bh * p.P * D;
  const bool rows8 = D == 128 && (p.P % (8 * nw)) == 0;   // N = 64: a state row is one float4 per lane
  float4 z[8];
  if (rows8) {
#pragma unroll
    for (int r = 0; r < 8; ++r) z[r] = reinterpret_cast<const float4*>(state + (size_t)(8 * w + r) * D)[lane];
  }
  const bool one_pass = p.P <= (int)blockDim.x && p.N <= 64;   // one channel / one b pair per thread
  const T* convw = reinterpret_cast<const T*>(p.conv_w);
  float r_x = 0.f, r_bias = 0.f, r_win[3] = {0.f, 0.f, 0.f}, r_wgt[4] = {0.f, 0.f, 0.f, 0.f};
  float r_up = 0.f, r_gate = 0.f, r_dsk = 0.f, r_bp[2] = {0.f, 0.f}, r_bc[4] = {0.f, 0.f, 0.f, 0.f};
  if (one_pass) {
    if (tid < p.P) {
      const int c = h * p.P + tid;
      r_x = to_f32(reinterpret_cast<const T*>(p.value)[(size_t)b * p.value_stride + c]);
      r_gate = to_f32(reinterpret_cast<const T*>(p.gate)[(size_t)b * p.gate_stride + c]);
      r_up = to_f32(reinterpret_cast<const T*>(p.u_prev)[(size_t)bh * p.P + tid]);
      if (p.d_skip) r_dsk = p.d_skip[h];
      if (convw) {
        const T* st = reinterpret_cast<const T*>(p.conv_state) + ((size_t)b * C + c) * (p.W - 1);
        if (p.conv_b) r_bias = to_f32(reinterpret_cast<const T*>(p.conv_b)[c]);
        for (int j = 0; j < p.W - 1; ++j) r_win[j] = to_f32(st[j]);
        for (int j = 0; j < p.W; ++j) r_wgt[j] = to_f32(convw[(size_t)c * p.W + j]);
      }
    }
    if (w == 2 || w == 3) {
      const T* src = reinterpret_cast<const T*>(p.bc) + (size_t)b * p.bc_stride + (size_t)(4 * g + 2 * (w - 2)) * p.N;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int n = lane + 32 * q;
        if (n < p.N) { r_bc[2 * q] = to_f32(src[n]); r_bc[2 * q + 1] = to_f32(src[p.N + n]); }
      }
    }
    if (tid >= 128 && tid < 128 + p.N && p.b_prev_in) {   // (warps 4, 5: not the ones busy with b and c)
      const T* bpin = reinterpret_cast<const T*>(p.b_prev_in) + bg * D + 2 * (tid - 128);
      r_bp[0] = to_f32(bpin[0]); r_bp[1] = to_f32(bpin[1]);
    }
  }

  // ---- A. conv update of this head's channels ------------------------------------------------
  if (one_pass) {
    if (tid < p.P) {
      const int c = h * p.P + tid;
      float u = r_x;
      if (convw) {
        T* st = reinterpret_cast<T*>(p.conv_state) + ((size_t)b * C + c) * (p.W - 1);
        float a = r_bias;
        for (int j = 0; j < p.W - 1; ++j) a += r_wgt[j] * r_win[j];
        a += r_wgt[p.W - 1] * r_x;
        u = round_io<T>(silu_f(a));
        for (int j = 0; j + 1 < p.W - 1; ++j) st[j] = from_f32<T>(r_win[j + 1]);
        if (p.W > 1) st[p.W - 2] = from_f32<T>(r_x);
      }
      s_u[tid] = u;
      s_up[tid] = r_up;
      reinterpret_cast<T*>(p.u_prev)[(size_t)bh * p.P + tid] = from_f32<T>(u);
    }
  } else {
    for (int pp = tid; pp < p.P; pp += blockDim.x) {
      const int c = h * p.P + pp;
      T* st = reinterpret_cast<T*>(p.conv_state) + ((size_t)b * C + c) * (p.W - 1);
      const float x = to_f32(reinterpret_cast<const T*>(p.value)[(size_t)b * p.value_stride + c]);
      float u = x;
      if (convw) {
        float a = p.conv_b ? to_f32(reinterpret_cast<const T*>(p.conv_b)[c]) : 0.f;
        float win[4] = {0.f, 0.f, 0.f, 0.f};      // the carried inputs, oldest first
        for (int j = 0; j < p.W - 1; ++j) { win[j] = to_f32(st[j]); a += to_f32(convw[(size_t)c * p.W + j]) * win[j]; }
        a += to_f32(convw[(size_t)c * p.W + p.W - 1]) * x;
        u = round_io<T>(silu_f(a));
        for (int j = 0; j + 1 < p.W - 1; ++j) st[j] = from_f32<T>(win[j + 1]);
        if (p.W > 1) st[p.W - 2] = from_f32<T>(x);
      }
      T* up = reinterpret_cast<T*>(p.u_prev) + (size_t)bh * p.P + pp;
      s_u[pp] = u;
      s_up[pp] = to_f32(*up);
      *up = from_f32<T>(u);
    }
  }
  // ---- B. transition and taps of this head (one thread; float64 inside) ------------------------
  if (tid == blockDim.x - 1) {
    const T* pr = reinterpret_cast<const T*>(p.params) + (size_t)b * p.params_stride + 3 * h;
    const CoeffOut o = coeff_eval<false>(to_f32(pr[0]) + p.dt_bias[h], to_f32(pr[1]) + p.alpha_bias[h],
                                  to_f32(pr[2]) + p.theta_mod_bias[h], p.theta_bias[h], p.theta_sign[h], p.cfg);
    const zc kp = {o.dt * o.k2.re, o.dt * o.k2.im};
    s_coef[0] = (float)o.rho.re; s_coef[1] = (float)o.rho.im;
    s_coef[2] = (float)kp.re; s_coef[3] = (float)kp.im;
    s_coef[4] = (float)(o.dt * o.k1.re - kp.re); s_coef[5] = (float)(o.dt * o.k1.im - kp.im);
  }
  // ---- C. b and c of this head's group (warps 2, 3: one each) ------------------------------------
  if (w == 2 || w == 3) {
    const int which = w - 2;      // 0: b (rows 0, 1 of bc), 1: c (rows 2, 3)
    const T* src = reinterpret_cast<const T*>(p.bc) + (size_t)b * p.bc_stride + (size_t)(4 * g + 2 * which) * p.N;
    float* dst = which ? s_c : s_b;
    float ss = 0.f;
    if (one_pass) {
      float amp[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        amp[q] = lane + 32 * q < p.N ? softplus_f(r_bc[2 * q]) : 0.f;
        ss += amp[q] * amp[q];
      }
      ss = warp_sum(ss);
      const float inv = rsqrtf(fmaxf(ss / (float)p.N, p.cfg.eps));
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int n = lane + 32 * q;
        if (n < p.N) {
          float sn, cs;
          sincosf(3.14159265358979323846f * tanhf(r_bc[2 * q + 1]), &sn, &cs);
          dst[2 * n] = round_io<T>(amp[q] * inv * cs);
          dst[2 * n + 1] = round_io<T>(amp[q] * inv * sn);
        }
      }
    } else {
      for (int n = lane; n < p.N; n += 32) { const float a = softplus_f(to_f32(src[n])); ss += a * a; }
      ss = warp_sum(ss);
      const float inv = rsqrtf(fmaxf(ss / (float)p.N, p.cfg.eps));
      for (int n = lane; n < p.N; n += 32) {
        const float a = softplus_f(to_f32(src[n])) * inv;
        const float ph = 3.14159265358979323846f * tanhf(to_f32(src[p.N + n]));
        float sn, cs;
        sincosf(ph, &sn, &cs);
        dst[2 * n] = round_io<T>(a * cs);
        dst[2 * n + 1] = round_io<T>(a * sn);
      }
    }
  }
  __syncthreads();
  // ---- D. tap-weighted b vectors; the group's first head hands b on as the next token's b_prev ----
  {
    const cf kp = {s_coef[2], s_coef[3]}, kc = {s_coef[4], s_coef[5]};
    const T* bpin = reinterpret_cast<const T*>(p.b_prev_in);
    T* bpout = reinterpret_cast<T*>(p.b_prev_out);
    const bool hand_on = h % (p.H / p.G) == 0;
    auto taps = [&](int n, cf bp) {
      const cf bt = {s_b[2 * n], s_b[2 * n + 1]};
      const cf a = cmul(kp, bp), c2 = cmul(kc, bt);
      s_bp[2 * n] = a.re; s_bp[2 * n + 1] = a.im;
      s_bc[2 * n] = c2.re; s_bc[2 * n + 1] = c2.im;
      if (hand_on) { bpout[bg * D + 2 * n] = from_f32<T>(bt.re); bpout[bg * D + 2 * n + 1] = from_f32<T>(bt.im); }
    };
    if (one_pass) {
      if (tid >= 128 && tid < 128 + p.N) taps(tid - 128, cf{r_bp[0], r_bp[1]});
    } else {
      for (int n = tid; n < p.N; n += blockDim.x) {
        cf bp = {0.f, 0.f};
        if (bpin) bp = {to_f32(bpin[bg * D + 2 * n]), to_f32(bpin[bg * D + 2 * n + 1])};
        taps(n, bp);
      }
    }
  }
  __syncthreads();
  // ---- E. state update and read-out --------------------------------------------------------------
  const float mr = s_coef[0], mi = s_coef[1];
  if (rows8) {
    // a warp takes 8 rows at a time, all loads first (the first 8 were requested at the top)
    const float4 a = reinterpret_cast<const float4*>(s_bp)[lane];
    const float4 c = reinterpret_cast<const float4*>(s_bc)[lane];
    const float4 cc = reinterpret_cast<const float4*>(s_c)[lane];
    for (int p0 = 8 * w; p0 < p.P; p0 += 8 * nw) {
      if (p0 != 8 * w) {
#pragma unroll
        for (int r = 0; r < 8; ++r) z[r] = reinterpret_cast<const float4*>(state + (size_t)(p0 + r) * D)[lane];
      }
      float acc[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float u = s_u[p0 + r], up = s_up[p0 + r];
        float4 o;
        o.x = mr * z[r].x - mi * z[r].y + up * a.x + u * c.x;
        o.y = mr * z[r].y + mi * z[r].x + up * a.y + u * c.y;
        o.z = mr * z[r].z - mi * z[r].w + up * a.z + u * c.z;
        o.w = mr * z[r].w + mi * z[r].z + up * a.w + u * c.w;
        reinterpret_cast<float4*>(state + (size_t)(p0 + r) * D)[lane] = o;
        acc[r] = cc.x * o.x + cc.y * o.y + cc.z * o.z + cc.w * o.w;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) acc[r] = warp_sum(acc[r]);
      if (lane < 8) {
        float v = acc[0];
#pragma unroll
        for (int r = 1; r < 8; ++r) v = lane == r ? acc[r] : v;
        s_y[p0 + lane] = round_io<T>(v);
      }
    }
  } else {
    for (int pp = w; pp < p.P; pp += nw) {
      const float u = s_u[pp], up = s_up[pp];
      float* zr = state + (size_t)pp * D;
      float acc = 0.f;
      for (int n = lane; n < p.N; n += 32) {
        const float2 z = reinterpret_cast<const float2*>(zr)[n];
        float2 o;
        o.x = mr * z.x - mi * z.y + up * s_bp[2 * n] + u * s_bc[2 * n];
        o.y = mr * z.y + mi * z.x + up * s_bp[2 * n + 1] + u * s_bc[2 * n + 1];
        reinterpret_cast<float2*>(zr)[n] = o;
        acc += s_c[2 * n] * o.x + s_c[2 * n + 1] * o.y;
      }
      acc = warp_sum(acc);
      if (lane == 0) s_y[pp] = round_io<T>(acc);
    }
  }
  __syncthreads();
  // ---- F. skip, gate, partial sum of squares ------------------------------------------------------
  float ss = 0.f;
  for (int pp = tid; pp < p.P; pp += blockDim.x) {
    const int c = h * p.P + pp;
    float pre = s_y[pp];
    if (p.d_skip) pre = round_io<T>(pre + s_u[pp] * (one_pass ? r_dsk : p.d_skip[h]));
    const float gt = one_pass ? r_gate : to_f32(reinterpret_cast<const T*>(p.gate)[(size_t)b * p.gate_stride + c]);
    const float hv = round_io<T>(pre * silu_f(gt));
    reinterpret_cast<T*>(p.hid)[(size_t)b * C + c] = from_f32<T>(hv);
    ss += hv * hv;
  }
  ss = warp_sum(ss);
  if (lane == 0) p.part[(size_t)bh * 8 + w] = ss;   // (8 warps)
}

// ---- pipelined form: P = 64, 2N = 128 KQ ----------------------------------------------------------------------------
// Bound by the traffic of the float32 state (read once, written once).  One CTA per (batch, head) spent most of its
// life in the serial chain in front of the state update (conv, float64 coefficients, b and c, taps: ~10 us under load
// against the ~2 us its bytes take), so the work is cut into two groups of warps of a persistent CTA: five warps prepare
// the vectors of the NEXT (batch, head) while eight warps update the state of the current one.  A state warp owns 8
// rows (4 KB KQ, contiguous), keeps two loads and one store of them in flight as bulk copies through a ring of three
// tiles in shared memory, and needs no barrier with the other state warps.  Two CTAs per SM (KQ = 1) or one (KQ = 2)
// keep 128 KB of loads in flight per SM.
constexpr int STEP_WARPS = 8, PREP_WARPS = 5, STEP_RING = 3, STEP_THREADS = 32 * (STEP_WARPS + PREP_WARPS);
template <int KQ> struct StepSmem {
  static constexpr int D = 128 * KQ, TILE_FLOATS = 8 * D;
  static constexpr int VEC = 3 * D + 3 * 64 + 16;   // kp b_prev | kc b | c | u | u_prev | gate | m, kp, kc, d_skip
  static constexpr size_t BYTES = 4 * ((size_t)STEP_WARPS * STEP_RING * TILE_FLOATS + 2 * VEC) + 128;
};

template <typename T, int KQ>
__global__ void __launch_bounds__(STEP_THREADS, KQ == 1 ? 2 : 1) mixer_step_pipe_kernel(StepParams p, int tasks) {
  using SM = StepSmem<KQ>;
  using namespace tc;
  constexpr int D = SM::D, N = D / 2, P = 64, RC = 8 / KQ;   // RC rows at a time: 8 float4 per lane
  extern __shared__ __align__(128) float smem[];
  __shared__ uint64_t bar_tile[STEP_WARPS][STEP_RING], bar_full[2], bar_empty[2];
  __shared__ int s_abort;
  float* vecs = smem + STEP_WARPS * STEP_RING * SM::TILE_FLOATS;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, C = p.H * P;
  const int first = blockIdx.x, stride = gridDim.x, n = (tasks - first + stride - 1) / stride;   // this CTA's (batch, head)s
  if (tid == 0) {
    for (int i = 0; i < STEP_WARPS; ++i)
      for (int k = 0; k < STEP_RING; ++k) mbar_init(&bar_tile[i][k], 1);
    for (int k = 0; k < 2; ++k) { mbar_init(&bar_full[k], PREP_WARPS); mbar_init(&bar_empty[k], STEP_WARPS); }
    fence_barrier_init();
    s_abort = 0;
  }
  grid_release();
  __syncthreads();
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {   // a converged warp; bounded
    bool ok = mbar_try_wait(bar, parity);
    if (!ok) {
      const long long t0 = clock64();
      while (!(ok = mbar_try_wait(bar, parity))) {
        if (*reinterpret_cast<volatile int*>(&s_abort)) break;
        if (clock64() - t0 > WAIT_CLOCKS_DEFAULT) {
          atomicCAS(&g_step_status, 0, code);
          *reinterpret_cast<volatile int*>(&s_abort) = 1;
          break;
        }
      }
    }
    return __all_sync(0xffffffffu, ok) != 0;
  };

  if (w < STEP_WARPS) {
    // ---- state warps ------------------------------------------------------------------------------------------
    float* ring = smem + w * STEP_RING * SM::TILE_FLOATS;
    auto rows_of = [&](int j) { return p.state + ((size_t)(first + j * stride) * P + 8 * w) * D; };
    auto request = [&](int j) {   // lane 0
      mbar_expect_tx(&bar_tile[w][j % STEP_RING], SM::TILE_FLOATS * 4);
      bulk_load(ring + (j % STEP_RING) * SM::TILE_FLOATS, rows_of(j), SM::TILE_FLOATS * 4, &bar_tile[w][j % STEP_RING]);
    };
    int requested = min(n, 2);
    if (lane == 0)
      for (int j = 0; j < requested; ++j) request(j);
    bool live = true;
    for (int j = 0; j < n; ++j) {
      if (live && j + 2 < n) {   // the tile refilled here was stored in the previous iteration
        if (lane == 0) { tma_store_wait_read(); request(j + 2); }
        ++requested;
      }
      const int bh = first + j * stride, b = bh / p.H, h = bh % p.H;
      const float* v = vecs + (j & 1) * SM::VEC;
      const float *s_u = v + 3 * D, *s_up = s_u + P, *s_g = s_up + P, *s_coef = s_g + P;
      live = live && wait(&bar_full[j & 1], (j >> 1) & 1, 41);
      live = live && wait(&bar_tile[w][j % STEP_RING], (j / STEP_RING) & 1, 42);
      float ss = 0.f;
      if (live) {
        float* tile = ring + (j % STEP_RING) * SM::TILE_FLOATS;
        float4 a[KQ], c[KQ], cc[KQ];
#pragma unroll
        for (int q = 0; q < KQ; ++q) {
          a[q] = reinterpret_cast<const float4*>(v)[lane + 32 * q];
          c[q] = reinterpret_cast<const float4*>(v + D)[lane + 32 * q];
          cc[q] = reinterpret_cast<const float4*>(v + 2 * D)[lane + 32 * q];
        }
        const float mr = s_coef[0], mi = s_coef[1], dsk = s_coef[6];
#pragma unroll
        for (int r0 = 0; r0 < 8; r0 += RC) {
          float acc[RC];
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            const float u = s_u[8 * w + r0 + r], up = s_up[8 * w + r0 + r];
            acc[r] = 0.f;
#pragma unroll
            for (int q = 0; q < KQ; ++q) {
              float4* cell = reinterpret_cast<float4*>(tile + (r0 + r) * D) + lane + 32 * q;
              const float4 z = *cell;
              float4 o;
              o.x = mr * z.x - mi * z.y + up * a[q].x + u * c[q].x;
              o.y = mr * z.y + mi * z.x + up * a[q].y + u * c[q].y;
              o.z = mr * z.z - mi * z.w + up * a[q].z + u * c[q].z;
              o.w = mr * z.w + mi * z.z + up * a[q].w + u * c[q].w;
              *cell = o;
              acc[r] += cc[q].x * o.x + cc[q].y * o.y + cc[q].z * o.z + cc[q].w * o.w;
            }
          }
          // sum over the lanes, halving the rows a lane still holds at every step
#pragma unroll
          for (int half = RC / 2, o = 16; half >= 1; half >>= 1, o >>= 1) {
            const bool hi = (lane & o) != 0;
#pragma unroll
            for (int r = 0; r < half; ++r) {
              const float send = hi ? acc[r] : acc[r + half], keep = hi ? acc[r + half] : acc[r];
              acc[r] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          float y = acc[0];
#pragma unroll
          for (int o = 16 / RC; o >= 1; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
          // lane 32 / RC * r holds row r: skip, gate
          const int r = lane / (32 / RC), pp = 8 * w + r0 + r;
          if (lane % (32 / RC) == 0) {
            float pre = round_io<T>(y);
            if (p.d_skip) pre = round_io<T>(pre + s_u[pp] * dsk);
            const float hv = round_io<T>(pre * silu_f(s_g[pp]));
            reinterpret_cast<T*>(p.hid)[(size_t)b * C + h * P + pp] = from_f32<T>(hv);
            ss += hv * hv;
          }
        }
        ss = warp_sum(ss);
        fence_async_smem();
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bar_empty[j & 1]);
        if (live) {
          bulk_store(rows_of(j), ring + (j % STEP_RING) * SM::TILE_FLOATS, SM::TILE_FLOATS * 4);
          tma_store_commit();
          p.part[(size_t)bh * 8 + w] = ss;
        }
      }
    }
    if (lane == 0) {
      if (s_abort)   // loads in flight land before shared memory is released
        for (int j = max(0, requested - STEP_RING); j < requested; ++j) mbar_wait(&bar_tile[w][j % STEP_RING], (j / STEP_RING) & 1);
      tma_store_wait_all();
    }
  } else {
    // ---- preparation warps, one (batch, head) ahead: 8, 9 conv | 10 b and taps | 11 c | 12 coefficients ---------------
    grid_wait();   // the state tiles are already on their way
    const int pw = w - STEP_WARPS;
    bool live = true;
    for (int j = 0; j < n; ++j) {
      const int bh = first + j * stride, b = bh / p.H, h = bh % p.H, g = h / (p.H / p.G);
      const size_t bg = (size_t)b * p.G + g;
      float* v = vecs + (j & 1) * SM::VEC;
      float *s_u = v + 3 * D, *s_up = s_u + P, *s_g = s_up + P, *s_coef = s_g + P;
      if (pw < 2) {
        const int pp = 32 * pw + lane, c = h * P + pp;
        const T* convw = reinterpret_cast<const T*>(p.conv_w);
        const float x = to_f32(reinterpret_cast<const T*>(p.value)[(size_t)b * p.value_stride + c]);
        const float gate = to_f32(reinterpret_cast<const T*>(p.gate)[(size_t)b * p.gate_stride + c]);
        T* up_cell = reinterpret_cast<T*>(p.u_prev) + (size_t)bh * P + pp;
        const float up = to_f32(*up_cell);
        float u = x;
        if (convw) {
          T* st = reinterpret_cast<T*>(p.conv_state) + ((size_t)b * C + c) * (p.W - 1);
          float win[3] = {0.f, 0.f, 0.f}, wgt[4] = {0.f, 0.f, 0.f, 0.f};
          float a = p.conv_b ? to_f32(reinterpret_cast<const T*>(p.conv_b)[c]) : 0.f;
#pragma unroll
          for (int q = 0; q < 3; ++q) if (q < p.W - 1) win[q] = to_f32(st[q]);
#pragma unroll
          for (int q = 0; q < 4; ++q) if (q < p.W) wgt[q] = to_f32(convw[(size_t)c * p.W + q]);
#pragma unroll
          for (int q = 0; q < 3; ++q) if (q < p.W - 1) a += wgt[q] * win[q];
          a += (p.W == 4 ? wgt[3] : p.W == 3 ? wgt[2] : p.W == 2 ? wgt[1] : wgt[0]) * x;
          u = round_io<T>(silu_f(a));
#pragma unroll
          for (int q = 0; q < 3; ++q) if (q < p.W - 1) st[q] = from_f32<T>(q + 1 < p.W - 1 ? win[q + 1 > 2 ? 2 : q + 1] : x);
        }
        *up_cell = from_f32<T>(u);
        if (j >= 2) live = live && wait(&bar_empty[j & 1], ((j >> 1) - 1) & 1, 43);
        if (live) { s_u[pp] = u; s_up[pp] = up; s_g[pp] = gate; }
      } else if (pw < 4) {
        const T* src = reinterpret_cast<const T*>(p.bc) + (size_t)b * p.bc_stride + (size_t)(4 * g + 2 * (pw - 2)) * N;
        float am[2 * KQ], ph[2 * KQ], ss = 0.f;
#pragma unroll
        for (int q = 0; q < 2 * KQ; ++q) { am[q] = to_f32(src[lane + 32 * q]); ph[q] = to_f32(src[N + lane + 32 * q]); }
        cf bp[2 * KQ];
        if (pw == 2) {
          const T* bpin = reinterpret_cast<const T*>(p.b_prev_in);
#pragma unroll
          for (int q = 0; q < 2 * KQ; ++q) {
            bp[q] = {0.f, 0.f};
            if (bpin) bp[q] = {to_f32(bpin[bg * D + 2 * (lane + 32 * q)]), to_f32(bpin[bg * D + 2 * (lane + 32 * q) + 1])};
          }
        }
#pragma unroll
        for (int q = 0; q < 2 * KQ; ++q) { am[q] = softplus_f(am[q]); ss += am[q] * am[q]; }
        ss = warp_sum(ss);
        const float inv = rsqrtf(fmaxf(ss / (float)N, p.cfg.eps));
        cf bc[2 * KQ];
#pragma unroll
        for (int q = 0; q < 2 * KQ; ++q) {
          float sn, cs;
          sincosf(3.14159265358979323846f * tanhf(ph[q]), &sn, &cs);
          bc[q] = {round_io<T>(am[q] * inv * cs), round_io<T>(am[q] * inv * sn)};
        }
        if (j >= 2) live = live && wait(&bar_empty[j & 1], ((j >> 1) - 1) & 1, 43);
        if (pw == 3) {
          if (live) {
#pragma unroll
            for (int q = 0; q < 2 * KQ; ++q) reinterpret_cast<float2*>(v + 2 * D)[lane + 32 * q] = make_float2(bc[q].re, bc[q].im);
          }
        } else {
          bar_sync(1, 64);   // the coefficients of this (batch, head)
          const cf kp = {s_coef[2], s_coef[3]}, kc = {s_coef[4], s_coef[5]};
          if (live) {
            T* bpout = reinterpret_cast<T*>(p.b_prev_out) + bg * D;
            const bool hand_on = h % (p.H / p.G) == 0;   // the group's first head hands b on as the next token's b_prev
#pragma unroll
            for (int q = 0; q < 2 * KQ; ++q) {
              const cf x = cmul(kp, bp[q]), y = cmul(kc, bc[q]);
              reinterpret_cast<float2*>(v)[lane + 32 * q] = make_float2(x.re, x.im);
              reinterpret_cast<float2*>(v + D)[lane + 32 * q] = make_float2(y.re, y.im);
              if (hand_on) { bpout[2 * (lane + 32 * q)] = from_f32<T>(bc[q].re); bpout[2 * (lane + 32 * q) + 1] = from_f32<T>(bc[q].im); }
            }
          }
        }
      } else {
        const T* pr = reinterpret_cast<const T*>(p.params) + (size_t)b * p.params_stride + 3 * h;
        const CoeffOut o = coeff_eval<false>(to_f32(pr[0]) + p.dt_bias[h], to_f32(pr[1]) + p.alpha_bias[h],
                                             to_f32(pr[2]) + p.theta_mod_bias[h], p.theta_bias[h], p.theta_sign[h], p.cfg);
        const zc kp = {o.dt * o.k2.re, o.dt * o.k2.im};
        const float dsk = p.d_skip ? p.d_skip[h] : 0.f;
        if (j >= 2) live = live && wait(&bar_empty[j & 1], ((j >> 1) - 1) & 1, 43);
        if (lane == 0) {
          s_coef[0] = (float)o.rho.re; s_coef[1] = (float)o.rho.im;
          s_coef[2] = (float)kp.re; s_coef[3] = (float)kp.im;
          s_coef[4] = (float)(o.dt * o.k1.re - kp.re); s_coef[5] = (float)(o.dt * o.k1.im - kp.im);
          s_coef[6] = dsk;
        }
        bar_sync(1, 64);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_full[j & 1]);
    }
  }
}

// normed = hid * rsqrt(mean hid^2 + eps) * w, one CTA per batch row
template <typename T>
__global__ void __launch_bounds__(256) step_norm_kernel(const T* __restrict__ hid, const float* __restrict__ part,
                                                        const T* __restrict__ w, T* __restrict__ out, int C, int parts,
                                                        float eps) {
  __shared__ float s_red[8];
  const int b = blockIdx.x, lane = threadIdx.x & 31;
  float ss = 0.f;
  for (int k = threadIdx.x; k < parts; k += 256) ss += part[(size_t)b * parts + k];
  ss = warp_sum(ss);
  if (lane == 0) s_red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) tot += s_red[k];
  const float rstd = rsqrtf(tot / (float)C + eps);
  for (int c = threadIdx.x; c < C; c += 256) out[(size_t)b * C + c] = from_f32<T>(to_f32(hid[(size_t)b * C + c]) * rstd * to_f32(w[c]));
}
}  // namespace

// workspace: hid (batch, C) in the io type | part (batch, H, 8)
size_t mixer_step_workspace(int batch, int heads, int P) {
  return round_up((size_t)batch * heads * P * 4, 256) + round_up((size_t)batch * heads * 32, 256);
}

// The site code of the first expired wait of the pipelined step on the current device (0 = none).
int mixer_step_device_status(bool reset) {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_step_status, sizeof(int));
  if (reset && v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_step_status, &zero, sizeof(int));
  }
  return v;
}

namespace {
template <typename T, int KQ>
int launch_step_pipe(const StepParams& p, int tasks, bool dependent, cudaStream_t st) {
  auto k = mixer_step_pipe_kernel<T, KQ>;
  static std::atomic<unsigned long long> done{0};
  if (int e = ensure_smem(k, StepSmem<KQ>::BYTES, done)) return e;
  const int resident = 148 * (KQ == 1 ? 2 : 1);   // persistent: as many CTAs as fit, tasks dealt out round robin
  if (int e = launch_chained(k, (unsigned)(tasks < resident ? tasks : resident), STEP_THREADS, StepSmem<KQ>::BYTES, st, dependent, p, tasks))
    return e;
  return SL_OK;
}
}  // namespace

int mixer_step_launch(const MixerStepArgs& a, cudaStream_t st) {
  if (!a.gate || !a.value || !a.params || !a.bc || !a.dt_bias || !a.alpha_bias || !a.theta_mod_bias || !a.theta_bias ||
      !a.theta_sign || !a.cfg || !a.state || !a.b_prev_out || !a.u_prev)
    return SL_ERR_NULL_POINTER;
  if (a.conv_weight && a.d_conv > 1 && !a.conv_state) return SL_ERR_NULL_POINTER;
  if (a.batch < 1 || a.heads < 1 || a.groups < 1 || a.heads % a.groups || a.P < 1 || a.N < 1 || a.d_conv < 1 || a.d_conv > 4)
    return SL_ERR_BAD_SHAPE;
  if (!dtype_ok(a.io_dtype)) return SL_ERR_UNSUPPORTED;
  if (!aligned(a.state, 16)) return SL_ERR_BAD_ALIGNMENT;
  if (!a.workspace || a.workspace_bytes < mixer_step_workspace(a.batch, a.heads, a.P)) return SL_ERR_WORKSPACE_TOO_SMALL;
  StepParams p{};
  p.gate = a.gate; p.value = a.value; p.gate_stride = a.gate_stride; p.value_stride = a.value_stride;
  p.params = a.params; p.bc = a.bc; p.params_stride = a.params_stride; p.bc_stride = a.bc_stride;
  p.conv_w = a.conv_weight; p.conv_b = a.conv_bias; p.conv_state = a.conv_state;
  p.dt_bias = a.dt_bias; p.alpha_bias = a.alpha_bias; p.theta_mod_bias = a.theta_mod_bias; p.theta_bias = a.theta_bias;
  p.theta_sign = a.theta_sign; p.d_skip = a.d_skip; p.cfg = *a.cfg;
  p.state = a.state; p.b_prev_in = a.b_prev_in; p.b_prev_out = a.b_prev_out; p.u_prev = a.u_prev;
  p.hid = a.workspace;
  p.part = step_partials(a.workspace, a.batch, a.heads, a.P);
  p.batch = a.batch; p.H = a.heads; p.G = a.groups; p.P = a.P; p.N = a.N; p.W = a.conv_weight ? a.d_conv : 1;
  const int tasks = a.batch * a.heads;
  // The pipelined form covers the head and state sizes whose rows are whole float4 per lane; others take one CTA per
  // (batch, head).
  if (a.P == 64 && (a.N == 64 || a.N == 128)) {
    int rc = SL_OK;
    SL_DISPATCH_DTYPE(a.io_dtype, T, { rc = a.N == 64 ? launch_step_pipe<T, 1>(p, tasks, a.dependent, st) : launch_step_pipe<T, 2>(p, tasks, a.dependent, st); });
    if (rc != SL_OK) return rc;
  } else {
    const size_t smem = ((size_t)4 * 2 * a.N + 3 * (size_t)a.P) * sizeof(float);
    if (smem > 48 * 1024) return SL_ERR_UNSUPPORTED;
    SL_DISPATCH_DTYPE(a.io_dtype, T, { mixer_step_kernel<T><<<(unsigned)tasks, 256, smem, st>>>(p); });
  }
  note_launches(1);
  return launch_status();
}

int mixer_step_norm(const void* workspace, const void* norm_weight, float eps, void* normed, int batch, int heads, int P,
                    int io_dtype, cudaStream_t st) {
  const float* part = step_partials(const_cast<void*>(workspace), batch, heads, P);
  SL_DISPATCH_DTYPE(io_dtype, T, {
    step_norm_kernel<T><<<(unsigned)batch, 256, 0, st>>>(reinterpret_cast<const T*>(workspace), part,
                                                         reinterpret_cast<const T*>(norm_weight),
                                                         reinterpret_cast<T*>(normed), heads * P, heads * 8, eps);
  });
  note_launches(1);
  return launch_status();
}

}  // namespace sl

extern "C" size_t sl_mixer_decode_step_workspace_bytes(int batch, int heads, int P) {
  if (batch < 1 || heads < 1 || P < 1) return 0;
  return sl::mixer_step_workspace(batch, heads, P);
}

extern "C" int sl_mixer_decode_step(const void* gate, int64_t gate_row_stride, const void* value,
                                    int64_t value_row_stride, const void* params, const void* bc,
                                    const void* conv_weight, const void* conv_bias, void* conv_state,
                                    int d_conv, const float* dt_bias, const float* alpha_bias,
                                    const float* theta_mod_bias, const float* theta_bias,
                                    const float* theta_sign, const sl_scanprep_config* cfg,
                                    const float* d_skip, const void* norm_weight, float norm_eps,
                                    float* state, const void* b_prev_in, void* b_prev_out, void* u_prev,
                                    void* normed, void* workspace, size_t workspace_bytes, int batch,
                                    int heads, int groups, int P, int N, int io_dtype, void* stream) {
  using namespace sl;
  if (!norm_weight || !normed) return SL_ERR_NULL_POINTER;
  const MixerStepArgs a{gate, value, params, bc, gate_row_stride, value_row_stride, 3 * (int64_t)heads,
                        4 * (int64_t)groups * N, conv_weight, conv_bias, conv_state, d_conv, dt_bias, alpha_bias,
                        theta_mod_bias, theta_bias, theta_sign, cfg, d_skip, state, b_prev_in, b_prev_out, u_prev,
                        workspace, workspace_bytes, batch, heads, groups, P, N, io_dtype};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (int e = mixer_step_launch(a, st)) return e;
  return mixer_step_norm(workspace, norm_weight, norm_eps, normed, batch, heads, P, io_dtype, st);
}
