// Exact float32 sequential v2x2ssd scan (forward and backward), SIMT.
//
// This is the path taken for float32 inputs (parity to 1e-5 needs float32
// products, which the tensor cores do not offer) and for shapes the tensor-core
// path does not cover.  It evaluates the recurrence token by token exactly as the
// sequential oracle does (reference: slinoss/ops/v2x2ssd/reference.py:815-840):
//
//   z_t = m_t z_{t-1} + u_{t-1} (x) (kp_t b_{t-1}) + u_t (x) (kc_t b_t)
//   y_t[p] = Re sum_n conj(c_t[n]) z_t[p,n]
//
// One CTA owns one (batch, head, 64-row slice of P, segment of T).  A warp owns 32 rows of P and 4 NC complex columns of
// the state, a lane 4 rows of NC columns, kept in registers as packed pairs of columns for the whole segment.  With
// 8 x 4 lanes on the tile both sums (over columns for y, over rows for the gradients of b and c) are mostly inside a lane:
// 3 + 4 shuffles per token and warp, where a lane per row with all the columns needed 31 for every sum over rows.  Tokens
// are staged TB at a time in shared memory, already multiplied by their taps.
//
// Backward = two more sweeps of the same shape (in one launch: they do not depend on one another) plus two small
// finishing kernels:
//   sweep A (forward in time)  recomputes z_t and emits dc_t[n] = sum_p dy_t[p] z_t[p,n]
//   sweep B (backward in time) carries G_t = dy_t (x) c_t + conj(m_{t+1}) G_{t+1} and
//           emits dbc_t = sum_p u_t G_t, dbp_t = sum_p u_{t-1} G_t, dU, d_initial
//   finish  dK, dB, dC (group sums), and dM from the identity
//           conj(m_t) dm_t = S_t,  S_t = S_{t+1} + <c_t,dc_t> - conj(kp_t)dkp_t - conj(kc_t)dkc_t,
//           S_T = <d_final, z_final>   (no state history is needed for dM).
//
// The walk over T is serial, so a problem with few (batch, head) streams is split in time: a first launch runs every
// segment but the last from a zero state and keeps only where it ends and the product of its transitions; each CTA of the
// sweeps then folds the segments before its own into its start state (all in float32, the products in float64).  B the same,
// from the other end.  (2, 4, 256, P 64, N 32) forward + backward: 629 -> 74 us with 16 segments.
#include <algorithm>

#include "common.cuh"

namespace sl {
namespace {

struct SweepParams {
  const void *U, *B, *C, *Bprev, *Uprev, *dY;
  const float *M, *K, *z0, *dfinal;
  void* Y;
  float* zfinal;
  float *dc_head, *dbc_head, *dbp_head;  // (batch, heads, T, 2N) float32
  float* sT;                             // (batch, heads, 2)  <d_final, z_final>
  void *dU, *dUprev;
  float* dinit;
  float *zloc, *zprod, *gloc, *gprod;    // per segment: (batch, heads, P, 2N) end of the walk from zero, (batch, heads, 2)
  int batch, heads, groups, T, P, N;
  int NS, PW, TB, ptiles, nseg, seg_len;
};

// Sum over the lanes whose index differs in the bits HI .. LO (powers of two), scattering the values: a lane ends with LEN
// divided by as many halvings as there are bits, the others are plain sums.
template <int LEN, int HI, int LO>
struct Scatter {
  static __device__ __forceinline__ void run(float* v, int lane) {
    if constexpr (HI >= LO) {
      if constexpr (LEN > 1) {
        constexpr int H = LEN / 2;
        const bool up = (lane & HI) != 0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
          const float send = up ? v[i] : v[i + H], keep = up ? v[i + H] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, HI);
        }
        Scatter<H, HI / 2, LO>::run(v, lane);
      } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], HI);
        Scatter<1, HI / 2, LO>::run(v, lane);
      }
    }
  }
};

template <typename T>
__device__ __forceinline__ cf load_c(const T* base, size_t cidx) {
  return {to_f32(base[2 * cidx]), to_f32(base[2 * cidx + 1])};
}

// Where a thread sits: its warp's run of columns and rows, its 4 rows and NC columns (NC / 2 pairs).
template <int NC>
struct Place {
  int lane, w, ns, pw, rg, cg, pl, pair;   // pl: first of the 4 rows inside the CTA tile; pair: first column pair
  __device__ __forceinline__ Place(const SweepParams& p) {
    lane = threadIdx.x & 31; w = threadIdx.x >> 5;
    ns = w % p.NS; pw = w / p.NS; rg = lane >> 2; cg = lane & 3;
    pl = pw * 32 + rg * 4; pair = (ns * 4 + cg) * (NC / 2);
  }
};
// 4 rows x NC / 2 pairs of columns, real and imaginary parts
template <int NC> struct Tile { f2 re[4][NC / 2], im[4][NC / 2]; };

// src (P, 2N) of one (batch, head): the thread's piece, zeros outside
template <int NC>
__device__ __forceinline__ void load_tile(Tile<NC>& z, const float* src, const Place<NC>& o, int row0, int P, int N) {
  const bool whole = (N & 1) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;   // 2 columns as one 16-byte piece
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int i = 0; i < NC / 2; ++i) {
      const int n = 2 * (o.pair + i), row = row0 + r;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (src && row < P && n < N) {
        const float* q = src + (size_t)row * 2 * N + 2 * n;
        if (whole) v = *reinterpret_cast<const float4*>(q);
        else {
          v.x = q[0]; v.y = q[1];
          if (n + 1 < N) { v.z = q[2]; v.w = q[3]; }
        }
      }
      z.re[r][i] = mk2(v.x, v.z); z.im[r][i] = mk2(v.y, v.w);
    }
}
template <int NC>
__device__ __forceinline__ void store_tile(const Tile<NC>& z, float* dst, const Place<NC>& o, int row0, int P, int N) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int i = 0; i < NC / 2; ++i) {
      const int n = 2 * (o.pair + i), row = row0 + r;
      if (row >= P) continue;
      const float2 re = un2(z.re[r][i]), im = un2(z.im[r][i]);
      float* q = dst + (size_t)row * 2 * N + 2 * n;
      if (n < N) { q[0] = re.x; q[1] = im.x; }
      if (n + 1 < N) { q[2] = re.y; q[3] = im.y; }
    }
}
// z = m z + add (CONJ: conj(m) z + add)
template <int NC, bool CONJ>
__device__ __forceinline__ void advance_tile(Tile<NC>& z, float mr, float mi, const Tile<NC>& add) {
  const f2 r2 = dup2(mr), i2 = dup2(CONJ ? -mi : mi), n2 = dup2(CONJ ? mi : -mi);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int i = 0; i < NC / 2; ++i) {
      const f2 a = z.re[r][i], b = z.im[r][i];
      z.re[r][i] = fma2(n2, b, fma2(r2, a, add.re[r][i]));
      z.im[r][i] = fma2(i2, a, fma2(r2, b, add.im[r][i]));
    }
}
// Start state of a segment: the caller's state at that end of the sequence through the segments between, in walking order.
template <int NC, bool CONJ>
__device__ __forceinline__ void fold_tile(Tile<NC>& z, const SweepParams& p, const float* loc, const float* prod, int bh, int from,
                                          int step, int count, const Place<NC>& o, int row0) {
  const size_t bhs = (size_t)p.batch * p.heads;
  constexpr int DEPTH = 8 / NC;   // segments of a batch of loads
#pragma unroll 1
  for (int k = 0; k < count; k += DEPTH) {
    Tile<NC> add[DEPTH];
    float2 m[DEPTH];
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) {
      if (k + i >= count) continue;
      const size_t at = (from + step * (k + i)) * bhs + bh;
      m[i] = *reinterpret_cast<const float2*>(prod + 2 * at);
      load_tile<NC>(add[i], loc + at * p.P * 2 * p.N, o, row0, p.P, p.N);
    }
#pragma unroll
    for (int i = 0; i < DEPTH; ++i)
      if (k + i < count) advance_tile<NC, CONJ>(z, m[i].x, m[i].y, add[i]);
  }
}
// Product of the transitions [t0, t1) (1 past the end of the sequence), by one warp, to dst.
__device__ __forceinline__ void transition_product(const float* Mb, int t0, int t1, int T, float* dst) {
  const int lane = threadIdx.x & 31;
  double re = 1.0, im = 0.0;
  for (int t = t0 + lane; t < t1; t += 32) {
    if (t >= T) continue;
    const double mr = Mb[2 * t], mi = Mb[2 * t + 1], r = re * mr - im * mi;
    im = re * mi + im * mr; re = r;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double orr = __shfl_xor_sync(0xffffffffu, re, o), oi = __shfl_xor_sync(0xffffffffu, im, o);
    const double r = re * orr - im * oi;
    im = re * oi + im * orr; re = r;
  }
  if (lane == 0) { dst[0] = (float)re; dst[1] = (float)im; }
}

// What every sweep reads of one (batch, head, slice of P).
template <typename TIn, typename TY>
struct Stream {
  const TIn *U, *B, *C, *Bp, *Up;
  const TY* dY;
  const float *M, *K;
  int bh, row0, seg, t_lo, t_hi;   // row0: first row of the CTA tile; [t_lo, t_hi): the segment
  __device__ __forceinline__ Stream(const SweepParams& p, int pt, int segment) {
    const int h = blockIdx.x, b = blockIdx.y, g = h / (p.heads / p.groups), D = 2 * p.N;
    bh = b * p.heads + h;
    const int bg = b * p.groups + g;
    U = reinterpret_cast<const TIn*>(p.U) + (size_t)bh * p.T * p.P;
    B = reinterpret_cast<const TIn*>(p.B) + (size_t)bg * p.T * D;
    C = reinterpret_cast<const TIn*>(p.C) + (size_t)bg * p.T * D;
    Bp = p.Bprev ? reinterpret_cast<const TIn*>(p.Bprev) + (size_t)bg * D : nullptr;
    Up = p.Uprev ? reinterpret_cast<const TIn*>(p.Uprev) + (size_t)bh * p.P : nullptr;
    dY = p.dY ? reinterpret_cast<const TY*>(p.dY) + (size_t)bh * p.T * p.P : nullptr;
    M = p.M + (size_t)bh * p.T * 2;
    K = p.K + (size_t)bh * p.T * 4;
    row0 = pt * p.PW * 32; seg = segment;
    t_lo = seg * p.seg_len; t_hi = min(p.T, t_lo + p.seg_len);
  }
};

// A (rows, cols) array by the CTA, a warp per row: U rows are loaded, then stored, so that they cost one latency.
template <int U, typename V, typename Load, typename Store>
__device__ __forceinline__ void staged(int rows, int cols, Load load, Store store) {
  const int nw = blockDim.x >> 5;
#pragma unroll 1
  for (int c = threadIdx.x & 31; c < cols; c += 32)
#pragma unroll 1
    for (int r = threadIdx.x >> 5; r < rows; r += U * nw) {
      V v[U];
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (r + i * nw < rows) v[i] = load(r + i * nw, c);
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (r + i * nw < rows) store(r + i * nw, c, v[i]);
    }
}
template <typename F> __device__ __forceinline__ void each_row(int rows, int cols, F f) {
  for (int r = threadIdx.x >> 5; r < rows; r += blockDim.x >> 5)
    for (int c = threadIdx.x & 31; c < cols; c += 32) f(r, c);
}

// A token's columns in shared memory: pair (n, n+1) as re re im im
__device__ __forceinline__ int pair_slot(int n) { return 4 * (n >> 1) + (n & 1); }

// Stage tokens [t0, t0 + nb): the tapped b_{t-1} and b_t, c on request.
template <typename TIn, typename TY>
__device__ __forceinline__ void stage_columns(const SweepParams& p, const Stream<TIn, TY>& x, int t0, int nb, int Npad, float* s_bp,
                                              float* s_bc, float* s_c) {
  const int D = 2 * p.N, D2 = 2 * Npad;
  struct Piece { cf bt, bpv, ct; float4 k4; };
  staged<2, Piece>(nb, Npad, [&](int tt, int n) {
    const int t = t0 + tt;
    Piece v{};
    if (n < p.N) {
      if (s_bc) v.bt = load_c(x.B + (size_t)t * D, n);
      if (s_c) v.ct = load_c(x.C + (size_t)t * D, n);
      if (s_bp) {
        if (t > 0) v.bpv = load_c(x.B + (size_t)(t - 1) * D, n);
        else if (x.Bp) v.bpv = load_c(x.Bp, n);
      }
    }
    if (s_bp || s_bc) v.k4 = *reinterpret_cast<const float4*>(x.K + (size_t)t * 4);
    return v;
  }, [&](int tt, int n, const Piece& v) {
    const int o = tt * D2 + pair_slot(n);
    const cf bp = cmul({v.k4.x, v.k4.y}, v.bpv), bc = cmul({v.k4.z, v.k4.w}, v.bt);
    if (s_bp) { s_bp[o] = bp.re; s_bp[o + 2] = bp.im; }
    if (s_bc) { s_bc[o] = bc.re; s_bc[o + 2] = bc.im; }
    if (s_c) { s_c[o] = v.ct.re; s_c[o + 2] = v.ct.im; }
  });
}
// u of the tokens t0 - 1 .. t0 + nb - 1
template <typename TIn, typename TY>
__device__ __forceinline__ void stage_u(const SweepParams& p, const Stream<TIn, TY>& x, int t0, int nb, int PT, float* s_u) {
  staged<3, float>(nb + 1, PT, [&](int tt, int pp) {
    const int t = t0 + tt - 1, pr = x.row0 + pp;
    if (pr >= p.P) return 0.f;
    if (t >= 0) return to_f32(x.U[(size_t)t * p.P + pr]);
    return x.Up ? to_f32(x.Up[pr]) : 0.f;
  }, [&](int tt, int pp, float v) { s_u[tt * PT + pp] = v; });
}
template <typename TIn, typename TY>
__device__ __forceinline__ void stage_dy(const SweepParams& p, const Stream<TIn, TY>& x, int t0, int nb, int PT, float* s_dy) {
  staged<2, float>(nb, PT, [&](int tt, int pp) {
    const int pr = x.row0 + pp;
    return (pr < p.P && x.dY) ? to_f32(x.dY[(size_t)(t0 + tt) * p.P + pr]) : 0.f;
  }, [&](int tt, int pp, float v) { s_dy[tt * PT + pp] = v; });
}
// m of the tokens t0 + off ... (1 past the end of the sequence)
__device__ __forceinline__ void stage_m(const float* M, int t0, int nb, int T, float* s_m) {
  for (int idx = threadIdx.x; idx < nb; idx += blockDim.x) {
    const int t = t0 + idx;
    s_m[2 * idx] = t < T ? M[2 * (size_t)t] : 1.f;
    s_m[2 * idx + 1] = t < T ? M[2 * (size_t)t + 1] : 0.f;
  }
}

__device__ __forceinline__ void rows4(const float* s, f2 (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(s);
  v[0] = dup2(q.x); v[1] = dup2(q.y); v[2] = dup2(q.z); v[3] = dup2(q.w);
}
__device__ __forceinline__ void pair_at(const float* s, int pair, f2& re, f2& im) {
  const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(s + 4 * pair);
  re = q.x; im = q.y;
}
__device__ __forceinline__ float hsum(f2 v) { const float2 q = un2(v); return q.x + q.y; }
// sum over the rows of the warp of NC columns a lane: 2 NC values in smem order, scattered over the row lanes
template <int NC>
__device__ __forceinline__ void store_columns(const f2 (&re)[NC / 2], const f2 (&im)[NC / 2], int lane, int pair, float* dst) {
  float v[2 * NC];
#pragma unroll
  for (int i = 0; i < NC / 2; ++i) {
    const float2 a = un2(re[i]), b = un2(im[i]);
    v[4 * i] = a.x; v[4 * i + 1] = a.y; v[4 * i + 2] = b.x; v[4 * i + 3] = b.y;
  }
  Scatter<2 * NC, 16, 4>::run(v, lane);
  const int hi = (lane >> 4) & 1, mid = (lane >> 3) & 1, lo = (lane >> 2) & 1;
  if constexpr (NC == 2) {   // 4 values over 8 lanes: two lanes hold each
    if (!lo) dst[4 * pair + 2 * hi + mid] = v[0];
  } else {
    dst[4 * pair + 4 * hi + 2 * mid + lo] = v[0];
  }
}

// MODE 0: forward (writes Y, final state).  1: backward sweep A (writes dc_head, sT).  2: only where the segment ends.
template <typename TIn, typename TY, int NC, int MODE>
__device__ __forceinline__ void forward_sweep(const SweepParams& p, int pt, int seg, float* smem) {
  const Place<NC> o(p);
  const int NS = p.NS, PW = p.PW, TB = p.TB, Npad = NS * 4 * NC, D2 = 2 * Npad, PT = PW * 32, D = 2 * p.N, N = p.N, P = p.P;
  const Stream<TIn, TY> x(p, pt, seg);
  float* s_bp = smem;
  float* s_bc = s_bp + TB * D2;
  float* s_c = s_bc + TB * D2;
  float* s_u = s_c + TB * D2;             // (TB+1) x PT
  float* s_m = s_u + (TB + 1) * PT;       // TB x 2
  float* s_dy = s_m + 2 * TB;             // TB x PT       (MODE 1)
  float* s_part = s_dy + TB * PT;         // MODE0: TB x NS x PT ; MODE1: TB x PW x D2
  const int row0 = x.row0 + o.pl;

  Tile<NC> z;
  load_tile<NC>(z, MODE != 2 && p.z0 ? p.z0 + (size_t)x.bh * P * D : nullptr, o, row0, P, N);
  if (MODE != 2 && seg > 0) fold_tile<NC, false>(z, p, p.zloc, p.zprod, x.bh, 0, 1, seg, o, row0);
  if (MODE == 2 && pt == 0 && o.w == 0)
    transition_product(x.M, x.t_lo, x.t_hi, p.T, p.zprod + 2 * ((size_t)seg * p.batch * p.heads + x.bh));

  for (int t0 = x.t_lo; t0 < x.t_hi; t0 += TB) {
    const int nb = min(TB, x.t_hi - t0);
    stage_columns(p, x, t0, nb, Npad, s_bp, s_bc, MODE == 0 ? s_c : nullptr);
    stage_u(p, x, t0, nb, PT, s_u);
    if (MODE == 1) stage_dy(p, x, t0, nb, PT, s_dy);
    stage_m(x.M, t0, nb, p.T, s_m);
    __syncthreads();

    f2 up[4], u[4];
    rows4(s_u + o.pl, up);
#pragma unroll 1
    for (int tt = 0; tt < nb; ++tt) {
      const f2 mr = dup2(s_m[2 * tt]), mi = dup2(s_m[2 * tt + 1]), mn = dup2(-s_m[2 * tt + 1]);
      rows4(s_u + (tt + 1) * PT + o.pl, u);
      f2 acc[4], sre[NC / 2], sim[NC / 2], dy[4];
      if (MODE == 1) rows4(s_dy + tt * PT + o.pl, dy);
#pragma unroll
      for (int i = 0; i < NC / 2; ++i) {
        f2 ar, ai, cr, ci, qr, qi;
        pair_at(s_bp + tt * D2, o.pair + i, ar, ai);
        pair_at(s_bc + tt * D2, o.pair + i, cr, ci);
        if (MODE == 0) pair_at(s_c + tt * D2, o.pair + i, qr, qi);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f2 a = z.re[r][i], b = z.im[r][i];
          const f2 zr = fma2(u[r], cr, fma2(up[r], ar, fma2(mn, b, mul2(mr, a))));
          const f2 zi = fma2(u[r], ci, fma2(up[r], ai, fma2(mi, a, mul2(mr, b))));
          z.re[r][i] = zr; z.im[r][i] = zi;
          if (MODE == 0) acc[r] = fma2(qi, zi, i == 0 ? mul2(qr, zr) : fma2(qr, zr, acc[r]));
          if (MODE == 1) {
            sre[i] = r == 0 ? mul2(dy[r], zr) : fma2(dy[r], zr, sre[i]);
            sim[i] = r == 0 ? mul2(dy[r], zi) : fma2(dy[r], zi, sim[i]);
          }
        }
      }
      if (MODE == 0) {
        float v[4] = {hsum(acc[0]), hsum(acc[1]), hsum(acc[2]), hsum(acc[3])};
        Scatter<4, 2, 1>::run(v, o.lane);   // lane now holds row ``lane`` of the warp
        s_part[(tt * NS + o.ns) * PT + o.pw * 32 + o.lane] = v[0];
      }
      if (MODE == 1) store_columns<NC>(sre, sim, o.lane, o.pair, s_part + (tt * PW + o.pw) * D2);
#pragma unroll
      for (int r = 0; r < 4; ++r) up[r] = u[r];
    }
    __syncthreads();

    if (MODE == 0) {
      TY* Yb = reinterpret_cast<TY*>(p.Y) + (size_t)x.bh * p.T * P;
      each_row(nb, PT, [&](int tt, int pp) {
        const int pr = x.row0 + pp;
        if (pr < P) {
          float s = 0.f;
          for (int k = 0; k < NS; ++k) s += s_part[(tt * NS + k) * PT + pp];
          Yb[(size_t)(t0 + tt) * P + pr] = from_f32<TY>(s);
        }
      });
    }
    if (MODE == 1) {
      float* dcb = p.dc_head + (size_t)x.bh * p.T * D;
      each_row(nb, D, [&](int tt, int col) {
        const int slot = pair_slot(col >> 1) + 2 * (col & 1);
        float s = 0.f;
        for (int k = 0; k < PW; ++k) s += s_part[(tt * PW + k) * D2 + slot];
        float* dst = dcb + (size_t)(t0 + tt) * D + col;
        if (p.ptiles > 1) atomicAdd(dst, s); else *dst = s;
      });
    }
    // the staging of the next block only rewrites arrays last read before the
    // second barrier; s_part is next written after the first barrier of that block.
  }

  if (MODE == 2) store_tile<NC>(z, p.zloc + ((size_t)seg * p.batch * p.heads + x.bh) * P * D, o, row0, P, N);
  if (MODE == 0 && p.zfinal && seg == p.nseg - 1) store_tile<NC>(z, p.zfinal + (size_t)x.bh * P * D, o, row0, P, N);
  if (MODE == 1 && seg == p.nseg - 1) {
    // S_T = sum d_final * conj(z_final)
    Tile<NC> d;
    load_tile<NC>(d, p.dfinal ? p.dfinal + (size_t)x.bh * P * D : nullptr, o, row0, P, N);
    f2 sr2 = 0, si2 = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < NC / 2; ++i) {
        sr2 = fma2(d.re[r][i], z.re[r][i], fma2(d.im[r][i], z.im[r][i], sr2));
        si2 = add2(si2, fma2(d.im[r][i], z.re[r][i], mul2(mul2(d.re[r][i], dup2(-1.f)), z.im[r][i])));
      }
    const float sr = warp_sum(hsum(sr2)), si = warp_sum(hsum(si2));
    __syncthreads();
    if (o.lane == 0) { s_part[2 * o.w] = sr; s_part[2 * o.w + 1] = si; }
    __syncthreads();
    if (threadIdx.x == 0) {
      float ar = 0.f, ai = 0.f;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { ar += s_part[2 * k]; ai += s_part[2 * k + 1]; }
      float* dst = p.sT + (size_t)x.bh * 2;
      if (p.ptiles > 1) { atomicAdd(dst, ar); atomicAdd(dst + 1, ai); }
      else { dst[0] = ar; dst[1] = ai; }
    }
  }
}

// Backward sweep B: reverse in time.  STATES: only where the segment ends (at its first token).
template <typename TIn, typename TY, int NC, bool STATES>
__device__ __forceinline__ void reverse_sweep(const SweepParams& p, int pt, int seg, float* smem) {
  const Place<NC> o(p);
  const int NS = p.NS, PW = p.PW, TB = p.TB, Npad = NS * 4 * NC, D2 = 2 * Npad, PT = PW * 32, D = 2 * p.N, N = p.N, P = p.P;
  const Stream<TIn, TY> x(p, pt, seg);
  float* s_bp = smem;
  float* s_bc = s_bp + TB * D2;
  float* s_c = s_bc + TB * D2;
  float* s_u = s_c + TB * D2;              // (TB+1) x PT
  float* s_mn = s_u + (TB + 1) * PT;       // TB x 2 : m_{t+1}
  float* s_dy = s_mn + 2 * TB;             // TB x PT
  float* s_pc = s_dy + TB * PT;            // TB x PW x D2
  float* s_pp = s_pc + TB * PW * D2;       // TB x PW x D2
  float* s_duc = s_pp + TB * PW * D2;      // TB x NS x PT
  float* s_dup = s_duc + TB * NS * PT;     // TB x NS x PT
  float* s_carry = s_dup + TB * NS * PT;   // 2 x PT: what the token after a block adds to the block's last dU
  const int row0 = x.row0 + o.pl, t_last = (x.t_hi - x.t_lo - 1) / TB * TB + x.t_lo;

  Tile<NC> G;
  load_tile<NC>(G, !STATES && p.dfinal ? p.dfinal + (size_t)x.bh * P * D : nullptr, o, row0, P, N);
  if (!STATES && seg < p.nseg - 1)
    fold_tile<NC, true>(G, p, p.gloc, p.gprod, x.bh, p.nseg - 1, -1, p.nseg - 1 - seg, o, row0);
  if (STATES && pt == 0 && o.w == 0)
    transition_product(x.M, x.t_lo + 1, x.t_hi + 1, p.T, p.gprod + 2 * ((size_t)seg * p.batch * p.heads + x.bh));

  auto row_sums = [&](const f2 (&v)[4], float* dst) {   // over the lane's columns and the 4 column lanes
    float q[4] = {hsum(v[0]), hsum(v[1]), hsum(v[2]), hsum(v[3])};
    Scatter<4, 2, 1>::run(q, o.lane);
    dst[o.ns * PT + o.pw * 32 + o.lane] = q[0];
  };
  auto u_dot = [&](const float* s_col, f2 (&acc)[4]) {   // sum over the lane's columns of col . G
#pragma unroll
    for (int i = 0; i < NC / 2; ++i) {
      f2 cr, ci;
      pair_at(s_col, o.pair + i, cr, ci);
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r] = fma2(ci, G.im[r][i], i == 0 ? mul2(cr, G.re[r][i]) : fma2(cr, G.re[r][i], acc[r]));
    }
  };
  if (!STATES) {
    for (int idx = threadIdx.x; idx < 2 * PT; idx += blockDim.x) s_carry[idx] = 0.f;
    if (x.t_hi < p.T) {   // the token after the segment
      stage_columns(p, x, x.t_hi, 1, Npad, s_bp, static_cast<float*>(nullptr), static_cast<float*>(nullptr));
      __syncthreads();
      f2 acc[4];
      u_dot(s_bp, acc);
      row_sums(acc, s_dup);
      __syncthreads();
      for (int pp = threadIdx.x; pp < PT; pp += blockDim.x)
        for (int k = 0; k < NS; ++k) s_carry[pp] += s_dup[k * PT + pp];
      __syncthreads();
    }
  }

  int par = 0;
  for (int t0 = t_last; t0 >= x.t_lo; t0 -= TB, par ^= 1) {
    const int nb = min(TB, x.t_hi - t0);
    stage_columns(p, x, t0, nb, Npad, STATES ? nullptr : s_bp, STATES ? nullptr : s_bc, s_c);
    if (!STATES) stage_u(p, x, t0, nb, PT, s_u);
    stage_dy(p, x, t0, nb, PT, s_dy);
    stage_m(x.M, t0 + 1, nb, p.T, s_mn);
    __syncthreads();

#pragma unroll 1
    for (int tt = nb - 1; tt >= 0; --tt) {
      const f2 mr = dup2(s_mn[2 * tt]), mi = dup2(s_mn[2 * tt + 1]), mn = dup2(-s_mn[2 * tt + 1]);
      f2 dy[4];
      rows4(s_dy + tt * PT + o.pl, dy);
      // G = conj(m_{t+1}) G + dy * c_t
#pragma unroll
      for (int i = 0; i < NC / 2; ++i) {
        f2 qr, qi;
        pair_at(s_c + tt * D2, o.pair + i, qr, qi);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f2 a = G.re[r][i], b = G.im[r][i];
          G.re[r][i] = fma2(dy[r], qr, fma2(mi, b, mul2(mr, a)));
          G.im[r][i] = fma2(dy[r], qi, fma2(mn, a, mul2(mr, b)));
        }
      }
      if (STATES) continue;
      f2 acc[4], w[4], sre[NC / 2], sim[NC / 2];
      u_dot(s_bc + tt * D2, acc);
      row_sums(acc, s_duc + tt * NS * PT);
      u_dot(s_bp + tt * D2, acc);
      row_sums(acc, s_dup + tt * NS * PT);
      auto outer = [&](const float* s_row, float* dst) {
        rows4(s_row, w);
#pragma unroll
        for (int i = 0; i < NC / 2; ++i)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            sre[i] = r == 0 ? mul2(w[r], G.re[r][i]) : fma2(w[r], G.re[r][i], sre[i]);
            sim[i] = r == 0 ? mul2(w[r], G.im[r][i]) : fma2(w[r], G.im[r][i], sim[i]);
          }
        store_columns<NC>(sre, sim, o.lane, o.pair, dst);
      };
      outer(s_u + (tt + 1) * PT + o.pl, s_pc + (tt * PW + o.pw) * D2);
      outer(s_u + tt * PT + o.pl, s_pp + (tt * PW + o.pw) * D2);
    }
    __syncthreads();
    if (STATES) continue;

    each_row(nb, D, [&](int tt, int col) {
      const int slot = pair_slot(col >> 1) + 2 * (col & 1);
      float sc = 0.f, sp = 0.f;
      for (int k = 0; k < PW; ++k) {
        sc += s_pc[(tt * PW + k) * D2 + slot];
        sp += s_pp[(tt * PW + k) * D2 + slot];
      }
      const size_t q = ((size_t)x.bh * p.T + t0 + tt) * D + col;
      if (p.ptiles > 1) { atomicAdd(p.dbc_head + q, sc); atomicAdd(p.dbp_head + q, sp); }
      else { p.dbc_head[q] = sc; p.dbp_head[q] = sp; }
    });
    TIn* dUb = reinterpret_cast<TIn*>(p.dU) + (size_t)x.bh * p.T * P;
    each_row(nb, PT, [&](int tt, int pp) {
      const int pr = x.row0 + pp;
      float s = tt == nb - 1 ? s_carry[par * PT + pp] : 0.f;
      for (int k = 0; k < NS; ++k) s += s_duc[(tt * NS + k) * PT + pp];
      if (tt < nb - 1)
        for (int k = 0; k < NS; ++k) s += s_dup[((tt + 1) * NS + k) * PT + pp];
      if (pr < P) dUb[(size_t)(t0 + tt) * P + pr] = from_f32<TIn>(s);
      if (tt == 0) {
        float c = 0.f;
        for (int k = 0; k < NS; ++k) c += s_dup[k * PT + pp];
        s_carry[(par ^ 1) * PT + pp] = c;
      }
    });
    // the next block's staging rewrites arrays last read before the second barrier; s_pc, s_pp, s_duc, s_dup and the
    // other half of s_carry are next written or read after its first barrier.
  }
  if (STATES) {
    store_tile<NC>(G, p.gloc + ((size_t)seg * p.batch * p.heads + x.bh) * P * D, o, row0, P, N);
    return;
  }
  if (seg > 0) return;
  __syncthreads();
  if (p.dUprev) {
    TIn* dUp = reinterpret_cast<TIn*>(p.dUprev) + (size_t)x.bh * P;
    for (int pp = threadIdx.x; pp < PT; pp += blockDim.x)
      if (x.row0 + pp < P) dUp[x.row0 + pp] = from_f32<TIn>(s_carry[par * PT + pp]);
  }
  if (p.dinit) {
    Tile<NC> zero{};
    advance_tile<NC, true>(G, x.M[0], x.M[1], zero);
    store_tile<NC>(G, p.dinit + (size_t)x.bh * P * D, o, row0, P, N);
  }
}

// grid (heads, batch, ptiles x segments [x the two sweeps])
template <typename TIn, typename TY, int NC>
__global__ void __launch_bounds__(128 * NC) sweep_fwd_kernel(SweepParams p) {
  extern __shared__ __align__(16) float smem[];
  forward_sweep<TIn, TY, NC, 0>(p, blockIdx.z % p.ptiles, blockIdx.z / p.ptiles, smem);
}
template <typename TIn, typename TY, int NC>
__global__ void __launch_bounds__(128 * NC) sweep_bwd_kernel(SweepParams p) {
  extern __shared__ __align__(16) float smem[];
  const int pt = blockIdx.z % p.ptiles, seg = blockIdx.z / p.ptiles;   // the longer sweep first
  if (seg < p.nseg) reverse_sweep<TIn, TY, NC, false>(p, pt, seg, smem);
  else forward_sweep<TIn, TY, NC, 1>(p, pt, seg - p.nseg, smem);
}
// where each segment ends from zero: forward segments 0 .. nseg - 2, and for the backward also reverse segments 1 .. nseg - 1
template <typename TIn, typename TY, int NC>
__global__ void __launch_bounds__(128 * NC) segment_kernel(SweepParams p) {
  extern __shared__ __align__(16) float smem[];
  const int pt = blockIdx.z % p.ptiles, seg = blockIdx.z / p.ptiles;
  if (seg < p.nseg - 1) forward_sweep<TIn, TY, NC, 2>(p, pt, seg, smem);
  else reverse_sweep<TIn, TY, NC, true>(p, pt, seg - (p.nseg - 2), smem);
}

// One warp per (batch, group, t): dK and the dM scan terms per head, dB / dC summed
// over the heads of the group.
struct FinishParams {
  const void *B, *C, *Bprev;
  const float *K, *dc_head, *dbc_head, *dbp_head;
  float *dK, *sterm;
  void *dB, *dC, *dBprev;
  int batch, heads, groups, T, N;
};

template <typename TIn>
__global__ void __launch_bounds__(256) bwd_finish_kernel(FinishParams p) {
  constexpr int MAXN = 4;  // N <= 128
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long rows = (long long)p.batch * p.groups * p.T;
  if (row >= rows) return;
  const int t = (int)(row % p.T);
  const int bg = (int)(row / p.T);
  const int g = bg % p.groups, b = bg / p.groups;
  const int hpg = p.heads / p.groups, N = p.N, D = 2 * N, T = p.T;
  const TIn* Bb = reinterpret_cast<const TIn*>(p.B) + ((size_t)bg * T) * D;
  const TIn* Cb = reinterpret_cast<const TIn*>(p.C) + ((size_t)bg * T) * D;
  const TIn* Bp = p.Bprev ? reinterpret_cast<const TIn*>(p.Bprev) + (size_t)bg * D : nullptr;

  cf bt[MAXN], bprev[MAXN], ct[MAXN], db[MAXN], dc[MAXN], dbp0[MAXN];
#pragma unroll
  for (int i = 0; i < MAXN; ++i) {
    const int n = lane + 32 * i;
    bt[i] = bprev[i] = ct[i] = db[i] = dc[i] = dbp0[i] = {0.f, 0.f};
    if (n < N) {
      bt[i] = load_c(Bb + (size_t)t * D, n);
      ct[i] = load_c(Cb + (size_t)t * D, n);
      if (t > 0) bprev[i] = load_c(Bb + (size_t)(t - 1) * D, n);
      else if (Bp) bprev[i] = load_c(Bp, n);
    }
  }
  for (int hh = 0; hh < hpg; ++hh) {
    const int h = g * hpg + hh;
    const size_t bh = (size_t)b * p.heads + h;
    const float* Kt = p.K + (bh * T + t) * 4;
    const cf kp = {Kt[0], Kt[1]}, kc = {Kt[2], Kt[3]};
    cf kpn = {0.f, 0.f};
    if (t + 1 < T) kpn = {Kt[4], Kt[5]};
    const float* dch = p.dc_head + (bh * T + t) * D;
    const float* dbch = p.dbc_head + (bh * T + t) * D;
    const float* dbph = p.dbp_head + (bh * T + t) * D;
    float kcr = 0.f, kci = 0.f, kpr = 0.f, kpi = 0.f, sr = 0.f, si = 0.f;
#pragma unroll
    for (int i = 0; i < MAXN; ++i) {
      const int n = lane + 32 * i;
      if (n < N) {
        const cf vdc = {dch[2 * n], dch[2 * n + 1]};
        const cf vbc = {dbch[2 * n], dbch[2 * n + 1]};
        const cf vbp = {dbph[2 * n], dbph[2 * n + 1]};
        // dkc += dbc * conj(b_t); dkp += dbp * conj(b_{t-1}); s += c_t * conj(dc_t)
        kcr += vbc.re * bt[i].re + vbc.im * bt[i].im;
        kci += vbc.im * bt[i].re - vbc.re * bt[i].im;
        kpr += vbp.re * bprev[i].re + vbp.im * bprev[i].im;
        kpi += vbp.im * bprev[i].re - vbp.re * bprev[i].im;
        sr += ct[i].re * vdc.re + ct[i].im * vdc.im;
        si += ct[i].im * vdc.re - ct[i].re * vdc.im;
        db[i] = cadd(db[i], cmul_conj_a(kc, vbc));
        if (t + 1 < T) {
          const cf vbpn = {dbph[D + 2 * n], dbph[D + 2 * n + 1]};
          db[i] = cadd(db[i], cmul_conj_a(kpn, vbpn));
        }
        dc[i] = cadd(dc[i], vdc);
        if (t == 0) dbp0[i] = cadd(dbp0[i], cmul_conj_a(kp, vbp));
      }
    }
    kcr = warp_sum(kcr); kci = warp_sum(kci); kpr = warp_sum(kpr); kpi = warp_sum(kpi);
    sr = warp_sum(sr); si = warp_sum(si);
    if (lane == 0) {
      float* dKt = p.dK + (bh * T + t) * 4;
      dKt[0] = kpr; dKt[1] = kpi; dKt[2] = kcr; dKt[3] = kci;
      // s_t = <c,dc> - conj(kp) dkp - conj(kc) dkc
      const cf a = cmul_conj_a(kp, {kpr, kpi}), c2 = cmul_conj_a(kc, {kcr, kci});
      float* st = p.sterm + (bh * T + t) * 2;
      st[0] = sr - a.re - c2.re;
      st[1] = si - a.im - c2.im;
    }
  }
  TIn* dBo = reinterpret_cast<TIn*>(p.dB) + ((size_t)bg * T + t) * D;
  TIn* dCo = reinterpret_cast<TIn*>(p.dC) + ((size_t)bg * T + t) * D;
#pragma unroll
  for (int i = 0; i < MAXN; ++i) {
    const int n = lane + 32 * i;
    if (n < N) {
      dBo[2 * n] = from_f32<TIn>(db[i].re); dBo[2 * n + 1] = from_f32<TIn>(db[i].im);
      dCo[2 * n] = from_f32<TIn>(dc[i].re); dCo[2 * n + 1] = from_f32<TIn>(dc[i].im);
      if (t == 0 && p.dBprev) {
        TIn* o = reinterpret_cast<TIn*>(p.dBprev) + (size_t)bg * D;
        o[2 * n] = from_f32<TIn>(dbp0[i].re); o[2 * n + 1] = from_f32<TIn>(dbp0[i].im);
      }
    }
  }
}

// One CTA per (batch, head): S_t = S_T + sum_{s >= t} sterm_s ; dM_t = S_t / conj(m_t).
__global__ void __launch_bounds__(256) bwd_dm_scan_kernel(const float* __restrict__ sterm,
                                                          const float* __restrict__ sT,
                                                          const float* __restrict__ M,
                                                          float* __restrict__ dM, int T) {
  __shared__ double s_wr[8], s_wi[8];
  __shared__ double s_carry[2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const size_t bh = blockIdx.x;
  const float* st = sterm + bh * T * 2;
  const float* Mb = M + bh * T * 2;
  float* dMb = dM + bh * T * 2;
  if (tid == 0) { s_carry[0] = sT[bh * 2]; s_carry[1] = sT[bh * 2 + 1]; }
  __syncthreads();
  for (int hi = T; hi > 0; hi -= 256) {
    const int t = hi - 1 - tid;  // thread 0 owns the latest token of the tile
    double vr = 0.0, vi = 0.0;
    if (t >= 0) { vr = st[2 * t]; vi = st[2 * t + 1]; }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double ar = __shfl_up_sync(0xffffffffu, vr, o), ai = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) { vr += ar; vi += ai; }
    }
    if (lane == 31) { s_wr[w] = vr; s_wi[w] = vi; }
    __syncthreads();
    double offr = s_carry[0], offi = s_carry[1];
    for (int k = 0; k < w; ++k) { offr += s_wr[k]; offi += s_wi[k]; }
    vr += offr; vi += offi;
    if (t >= 0) {
      const float mr = Mb[2 * t], mi = Mb[2 * t + 1];
      const float den = mr * mr + mi * mi;
      // S / conj(m) = S * m / |m|^2
      float outr = 0.f, outi = 0.f;
      if (den > 0.f) {
        outr = (float)((vr * mr - vi * mi) / den);
        outi = (float)((vr * mi + vi * mr) / den);
      }
      dMb[2 * t] = outr; dMb[2 * t + 1] = outi;
    }
    __syncthreads();
    if (tid == 255) { s_carry[0] = vr; s_carry[1] = vi; }
    __syncthreads();
  }
}

constexpr size_t SIMT_SMEM_MAX = 200 * 1024;
struct SimtConfig {
  int NC, NS, PW, ptiles, TB, threads, nseg, seg_len;
  size_t smem_fwd, smem_rev;
};

// Segments of T.  Per token a CTA takes as long alone on its SM as with others up to 8 warps; a split adds a pre-pass (half
// the work of a sweep), its launch (worth about 30 tokens) and a fold of one per segment passed.  Sequences up to 64 tokens stay whole.
void plan_segments(const ScanDims& d, SimtConfig& c) {
  c.nseg = 1; c.seg_len = d.T;
  if (d.T <= 64) return;
  const double ctas = (double)d.batch * d.heads * c.ptiles, slots = 148.0 * std::max(1, 256 / c.threads);
  double best = d.T * std::max(1.0, ctas / slots);
  for (int n = 2; n <= 64; ++n) {
    const int len = ((d.T + n - 1) / n + c.TB - 1) / c.TB * c.TB, segs = (d.T + len - 1) / len;
    if (segs < 2) break;
    const double cost = 1.5 * len * std::max(1.0, ctas * segs / slots) + 30 + segs;
    if (cost < 0.9 * best || (cost < best && c.nseg > 1)) { best = cost; c.nseg = segs; c.seg_len = len; }
  }
}

bool make_config(const ScanDims& d, SimtConfig& c) {
  if (d.N < 1 || d.N > 128 || d.P < 1) return false;
  c.NC = d.N <= 32 ? 2 : 4;
  c.NS = (d.N + 4 * c.NC - 1) / (4 * c.NC);
  c.PW = d.P > 32 ? 2 : 1;
  const int PT = 32 * c.PW;
  c.ptiles = (d.P + PT - 1) / PT;
  c.threads = 32 * c.NS * c.PW;
  const int D2 = 2 * c.NS * 4 * c.NC;
  for (c.TB = 16; c.TB >= 4; c.TB /= 2) {
    const size_t TB = c.TB;
    const size_t part_fwd = TB * (size_t)std::max(c.NS * PT, c.PW * D2);
    c.smem_fwd = 4 * (3 * TB * D2 + (TB + 1) * PT + 2 * TB + TB * PT + part_fwd);
    c.smem_rev = 4 * (3 * TB * D2 + (TB + 1) * PT + 2 * TB + TB * PT + 2 * TB * c.PW * D2 +
                      2 * TB * c.NS * PT + 2 * PT);
    if (c.smem_rev <= SIMT_SMEM_MAX) { plan_segments(d, c); return true; }
  }
  return false;
}

SweepParams base_params(const void* U, const float* M, const float* K, const void* B,
                        const void* C, const float* z0, const void* Bprev, const void* Uprev,
                        const ScanDims& d, const SimtConfig& c) {
  SweepParams p{};
  p.U = U; p.B = B; p.C = C; p.Bprev = Bprev; p.Uprev = Uprev; p.M = M; p.K = K; p.z0 = z0;
  p.batch = d.batch; p.heads = d.heads; p.groups = d.groups; p.T = d.T; p.P = d.P; p.N = d.N;
  p.NS = c.NS; p.PW = c.PW; p.TB = c.TB; p.ptiles = c.ptiles; p.nseg = c.nseg; p.seg_len = c.seg_len;
  return p;
}

// scratch of one direction: where the segments end, and the products of their transitions
size_t segment_floats(const ScanDims& d, const SimtConfig& c) {
  if (c.nseg == 1) return 0;
  const size_t bh = (size_t)d.batch * d.heads;
  return round_up(c.nseg * bh * ((size_t)d.P * 2 * d.N + 2), 64);
}
void segment_scratch(const ScanDims& d, const SimtConfig& c, float* at, float** loc, float** prod) {
  *loc = at;
  *prod = at + (size_t)c.nseg * d.batch * d.heads * d.P * 2 * d.N;
}

template <typename TIn, typename TY, int NC>
int launch_sweeps(const SweepParams& p, const SimtConfig& c, bool bwd, cudaStream_t st) {
  auto pre = segment_kernel<TIn, TY, NC>;
  auto k = bwd ? sweep_bwd_kernel<TIn, TY, NC> : sweep_fwd_kernel<TIn, TY, NC>;
  const size_t smem = bwd ? c.smem_rev : c.smem_fwd;
  static std::atomic<unsigned long long> done[3];
  if (int e = ensure_smem(k, SIMT_SMEM_MAX, done[bwd])) return e;
  if (int e = c.nseg > 1 ? ensure_smem(pre, SIMT_SMEM_MAX, done[2]) : SL_OK) return e;
  const unsigned dirs = bwd ? 2 : 1;
  if (c.nseg > 1) {
    pre<<<dim3(p.heads, p.batch, dirs * (c.nseg - 1) * c.ptiles), c.threads, c.smem_fwd, st>>>(p);
    note_launches(1);
  }
  k<<<dim3(p.heads, p.batch, dirs * c.nseg * c.ptiles), c.threads, smem, st>>>(p);
  note_launches(1);
  return launch_status();
}

}  // namespace

bool scan_simt_supported(const ScanDims& d) {
  SimtConfig c;
  return make_config(d, c);
}

size_t scan_simt_fwd_workspace(const ScanDims& d) {
  SimtConfig c;
  return make_config(d, c) ? 4 * segment_floats(d, c) : 0;
}

// Without its workspace the sequence is walked whole.
int scan_simt_fwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                  const float* z0, const void* Bprev, const void* Uprev, void* Y, float* zfinal,
                  const ScanDims& d, int io_dtype, int y_dtype, void* ws, size_t ws_bytes, cudaStream_t st) {
  SimtConfig c;
  if (!make_config(d, c)) return SL_ERR_UNSUPPORTED;
  if (!ws || ws_bytes < 4 * segment_floats(d, c) || !aligned(ws, 16)) { c.nseg = 1; c.seg_len = d.T; }
  SweepParams p = base_params(U, M, K, B, C, z0, Bprev, Uprev, d, c);
  p.Y = Y; p.zfinal = zfinal;
  segment_scratch(d, c, reinterpret_cast<float*>(ws), &p.zloc, &p.zprod);
  int rc = SL_ERR_UNSUPPORTED;
  SL_DISPATCH_DTYPE(io_dtype, TIn, SL_DISPATCH_DTYPE(y_dtype, TY, {
    rc = c.NC == 2 ? launch_sweeps<TIn, TY, 2>(p, c, false, st) : launch_sweeps<TIn, TY, 4>(p, c, false, st);
  }));
  return rc;
}

// workspace layout: dc_head | dbc_head | dbp_head (each batch*heads*T*2N floats) |
//                   sterm (batch*heads*T*2) | sT (batch*heads*2) | the segments of the two sweeps
size_t scan_simt_bwd_workspace(const ScanDims& d) {
  const size_t bht = (size_t)d.batch * d.heads * d.T;
  return round_up(4 * (3 * bht * 2 * d.N + bht * 2 + (size_t)d.batch * d.heads * 2), 256);
}
size_t scan_simt_bwd_split_workspace(const ScanDims& d) {
  SimtConfig c;
  return scan_simt_bwd_workspace(d) + (make_config(d, c) ? 8 * segment_floats(d, c) : 0);
}

// With scan_simt_bwd_workspace() bytes the sequence is walked whole, with scan_simt_bwd_split_workspace() in segments.
int scan_simt_bwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                  const float* z0, const void* Bprev, const void* Uprev, const void* dY,
                  const float* dfinal, void* dU, float* dM, float* dK, void* dB, void* dC,
                  float* dinit, void* dBprev, void* dUprev, const ScanDims& d, int io_dtype,
                  int dy_dtype, void* ws, size_t ws_bytes, cudaStream_t st) {
  SimtConfig c;
  if (!make_config(d, c)) return SL_ERR_UNSUPPORTED;
  const size_t need = scan_simt_bwd_workspace(d);
  if (!ws || ws_bytes < need) return SL_ERR_WORKSPACE_TOO_SMALL;
  if (ws_bytes < need + 8 * segment_floats(d, c) || !aligned(ws, 16)) { c.nseg = 1; c.seg_len = d.T; }
  const size_t bht = (size_t)d.batch * d.heads * d.T, D = 2 * (size_t)d.N;
  float* dc_head = reinterpret_cast<float*>(ws);
  float* dbc_head = dc_head + bht * D;
  float* dbp_head = dbc_head + bht * D;
  float* sterm = dbp_head + bht * D;
  float* sT = sterm + bht * 2;
  if (c.ptiles > 1) {  // partial sums of the P tiles are accumulated atomically
    if (cudaMemsetAsync(ws, 0, need, st) != cudaSuccess) return SL_ERR_LAUNCH_FAILED;
  }
  SweepParams p = base_params(U, M, K, B, C, z0, Bprev, Uprev, d, c);
  p.dY = dY; p.dfinal = dfinal; p.dc_head = dc_head; p.dbc_head = dbc_head;
  p.dbp_head = dbp_head; p.sT = sT; p.dU = dU; p.dUprev = dUprev; p.dinit = dinit;
  float* segments = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + need);
  segment_scratch(d, c, segments, &p.zloc, &p.zprod);
  segment_scratch(d, c, segments + segment_floats(d, c), &p.gloc, &p.gprod);
  int rc = SL_ERR_UNSUPPORTED;
  SL_DISPATCH_DTYPE(io_dtype, TIn, SL_DISPATCH_DTYPE(dy_dtype, TY, {
    rc = c.NC == 2 ? launch_sweeps<TIn, TY, 2>(p, c, true, st) : launch_sweeps<TIn, TY, 4>(p, c, true, st);
  }));
  if (rc != SL_OK) return rc;
  FinishParams f{};
  f.B = B; f.C = C; f.Bprev = Bprev; f.K = K; f.dc_head = dc_head; f.dbc_head = dbc_head;
  f.dbp_head = dbp_head; f.dK = dK; f.sterm = sterm; f.dB = dB; f.dC = dC; f.dBprev = dBprev;
  f.batch = d.batch; f.heads = d.heads; f.groups = d.groups; f.T = d.T; f.N = d.N;
  const long long rows = (long long)d.batch * d.groups * d.T;
  const unsigned blocks = (unsigned)((rows + 7) / 8);
  SL_DISPATCH_DTYPE(io_dtype, TIn, { bwd_finish_kernel<TIn><<<blocks, 256, 0, st>>>(f); });
  bwd_dm_scan_kernel<<<d.batch * d.heads, 256, 0, st>>>(sterm, sT, M, dM, d.T);
  note_launches(2);
  return launch_status();
}

}  // namespace sl
