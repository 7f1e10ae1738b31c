// Float32 v2x2ssd scan (forward and backward).
//
// This is the path taken for float32 inputs (parity to 1e-5 needs float32 products, which one tensor-core product is not)
// and for shapes the tensor-core path does not cover.  It evaluates the recurrence (reference:
// slinoss/ops/v2x2ssd/reference.py:815-840)
//
//   z_t = m_t z_{t-1} + u_{t-1} (x) (kp_t b_{t-1}) + u_t (x) (kc_t b_t),    y_t[p] = Re sum_n conj(c_t[n]) z_t[p,n]
//
// as V_t = z_t - u_t (x) (kc_t b_t), the state before the token's own injection, which has ONE injection per token and
// needs no division, so that an exactly zero transition is computed through:
//
//   V_{t+1} = m_{t+1} V_t + u_t (x) (h_t b_t),   h_t = m_{t+1} kc_t + kp_{t+1}   (m_T = 1, kp_T = 0: V_T is the final state)
//   y_t     = Re <c_t, V_t> + u_t Re(conj(c_t) kc_t b_t)
//
// in chunks of L = 16 tokens.  With P(j, i) = m_{i+2} .. m_j (products of at most 16 float32 transitions) and V the state at
// the chunk's first token:
//
//   y_j  = Re sum conj(c_j) a_j V + sum_{i<j} Re(P(j,i) h_i d(j,i)) u_i + Re(kc_j d(j,j)) u_j,  a_j = P(j,-1), d(j,i) = <c_j, b_i>
//   V'   = a_L V + sum_i u_i (x) (P(L,i) h_i b_i)
//
// Two multiply-adds per (row, real column) and token for each of the two instead of eight and six for a walk token by token.
// The adjoint (lambda_t of V_t) walks the chunks the other way with the same products; X(j,i) = <dy_j, u_i>:
//
//   A, forward in time: dC_j = a_j sum_p dy_j V + sum_{i<j} X(j,i) P(j,i) h_i b_i + X(j,j) kc_j b_j
//   B, backward:        D_i = conj(P(L,i)) sum_p u_i lambda + sum_{j>i} X(j,i) conj(P(j,i)) c_j,
//                       dB_i = conj(h_i) D_i + X(i,i) conj(kc_i) c_i,  dh_i = <b_i, D_i>  (-> dK),
//                       dU_i = Re sum conj(P(L,i) h_i b_i) lambda + sum_{j>=i} S(j,i) dy_j,   S: the factors of u_i in y_j
//   dM from S_t = S_{t+1} + <c_t, dC_t without its last term> - conj(h_t) dh_t,  conj(m_t) dm_t = S_t - conj(kp_t) dkp_t,
//   S_T = <d_final, z_final>, in float64 by the finishing kernel (no state history is kept).
//
// The products run on the tensor cores as products of bfloat16 parts (mma.sync m16n8k16): a float32 is the sum of three, a
// 16-bit operand of one or two, and the products of parts down to 2^-24 are kept (see products()), at 8 times the FMA rate.
// One CTA owns one (batch, head, 64 rows of P, segment of T); a warp owns 16 complex columns x 64 rows of the state, in
// registers as accumulators, which serve as the operand of the next chunk's products as they are (sums over the rows of P) or
// through an 8 x 8 transposition in registers (over the columns).  The operands that belong to a warp's columns are made by
// the warp itself from the raw rows, which arrive by cp.async one chunk ahead in their own type; only the sums over all
// columns (Y, dU, d(j,i)) and the per-token scalars cross warps.  The chain of transition products is one warp's, one chunk
// ahead.
//
// What bounds it now: issue and latency at 12 warps per SM: 168 registers hold the state, its parts and the operands, and the
// backward spills 280 to 740 bytes beside them.  Forward + backward, us, against sweeps token by token on the FMA pipe: (16, 4, 2048,
// N 48 fp16) 2973 -> 663, to which the looks for values that are not finite add 3 and the sums kept apart 2 (see below); (2, 4, 256,
// N 32 fp32) 61 -> 51.
// Distance from float64 against those sweeps (2-norm, float32 operands, T 256 to 4096, by shape): Y 1.26..1.29e-7 -> 1.07..1.12e-7,
// dU 1.13..1.15e-7 -> 1.07..1.12e-7, dB 1.08..1.09e-7 -> 1.01..1.02e-7, dC 1.25..1.26e-7 -> 1.05..1.06e-7, dK 1.27..1.32e-7 ->
// 1.19..1.24e-7, dM a third nearer.
//
// The walk over T is serial, so a problem with few (batch, head) streams is split in time: a first launch runs every
// segment but the last from a zero state and keeps only where it ends and the product of its transitions (in float64), a second
// one combines them to the segments' start states.  The adjoint's the same, from the other end.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace sl {
namespace {

constexpr int L = 16;          // tokens of a chunk
constexpr int ROWS = 64;       // rows of P of a CTA
constexpr int TABW = 18;       // row pitch (complex) of the table of products

struct SweepParams {
  const void *U, *B, *C, *Bprev, *Uprev, *dY;
  const float *M, *K, *z0, *dfinal;
  void* Y;
  float* zfinal;
  float *dB_head, *dC_head, *dBprev_head;   // (batch, heads, T, 2N) float32 where heads or rows of P are still to be summed
  float* sterm;                             // (batch, heads, T, 2)  <c_t, dC_t without the diagonal>
  float* sT;                                // (batch, heads, 2)     <d_final, z_final>
  float *dK, *dM;
  void *dU, *dB, *dC, *dUprev, *dBprev;
  float* dinit;
  float *zloc, *zprod, *gloc, *gprod;       // per segment: (batch, heads, P, 2N) end of the walk from zero, (batch, heads, 2)
  int batch, heads, groups, T, P, N;
  int W, ptiles, nseg, seg_len;             // W: warps, 16 complex columns each
  int spread;                               // dB, dC, dB_prev go to the float32 buffers
};

// Sum over the lanes whose index differs in the bits HI .. LO (powers of two), scattering the values: a lane ends with LEN
// divided by as many halvings as there are bits, the others are plain sums.
template <int LEN, int HI, int LO>
struct Scatter {
  static __device__ __forceinline__ void run(float* v, int lane) {
    if constexpr (HI >= LO) {
      constexpr int H = LEN / 2;
      const bool up = (lane & HI) != 0;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const float send = up ? v[i] : v[i + H], keep = up ? v[i + H] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, HI);
      }
      Scatter<H, HI / 2, LO>::run(v, lane);
    }
  }
};

// row pitch in bytes of an array of rows in shared memory: an odd number of 16-byte pieces (no bank conflicts across rows)
__host__ __device__ constexpr int row_pitch(int bytes) { return ((bytes + 15) / 16 | 1) * 16; }

// ---- float32 as sums of bfloat16 ---------------------------------------------------------------------------------------
// Parts that hold a type exactly (float32: 24 bits in three parts of 8).
template <typename T> struct Parts { static constexpr int N = 3; };
template <> struct Parts<__nv_bfloat16> { static constexpr int N = 1; };
template <> struct Parts<__half> { static constexpr int N = 2; };
// w[k] = part k of the pair v.  A finite float32 above the largest bfloat16 (the first part stays at that one) is its three parts
// too; of an infinity, as of a NaN, a part is NaN and so is every product with it.
template <int NP>
__device__ __forceinline__ void split(f2 v, uint32_t (&w)[NP]) {
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const float2 x = un2(v);
    if (k == 0 && NP == 3) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(w[k]) : "f"(x.y), "f"(x.x));
    else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[k]) : "f"(x.y), "f"(x.x));
    if (k + 1 < NP) v = fma2(mk2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u)), dup2(-1.f), v);
  }
}
template <bool FIRST>
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (FIRST)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  else asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = A B over 16 terms, smallest products first (those of parts whose weights together are below 2^-24 are left out).  The
// tensor cores cut the bits of a sum off instead of rounding them: that is harmless for the small products, and the large
// ones are added up here over 16 terms at most; longer sums go through rounded float32 additions.  Measured against float64
// over normal operands: 4.8e-8 relative for 16 terms and 6.3e-8 for 64, where a chain of fmaf has 7.4e-8 and 1.5e-7.
// NT independent tiles at a time, a product of each in turn: a tensor-core operation waits for the one before it on its sum.
// APART: the first parts' product, whose 16 terms of 16 bits are nearly exact, starts from zero too and the others' sum is added
// to it by a rounded addition instead of being cut off under it.  Where a result is common to many others its error does not average
// out: with the products over the rows of P (X) and with the state so, dB came from 1.11e-7 to 1.02e-7 of float64 and dU from 1.16e-7 to
// 1.12e-7 (1.09e-7 and 1.15e-7 token by token), at 684 -> 686 us for (16, 4, 2048, N 48 fp16); all products so: 9.0e-8, 703 us.
template <int NT, int NA, int NB, bool APART = false, typename FA, typename FB>
__device__ __forceinline__ void products(float (&d)[NT][4], FA a, FB b) {
  constexpr int SUM = NA + NB - 2 < 2 ? NA + NB - 2 : 2, FIRST = SUM - (NB - 1) > 0 ? SUM - (NB - 1) : 0;
#pragma unroll
  for (int sum = SUM; sum >= 0; --sum)
#pragma unroll
    for (int i = 0; i < NA; ++i)
      if (sum - i >= 0 && sum - i < NB)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          if (sum == SUM && i == FIRST) {
            mma<true>(d[t], a(t)[i], b(t)[sum - i][0], b(t)[sum - i][1]);
          } else if (APART && sum == 0) {
            float e[4];
            mma<true>(e, a(t)[0], b(t)[0][0], b(t)[0][1]);
            const float2 u = un2(add2(mk2(e[0], e[1]), mk2(d[t][0], d[t][1]))), v = un2(add2(mk2(e[2], e[3]), mk2(d[t][2], d[t][3])));
            d[t][0] = u.x; d[t][1] = u.y; d[t][2] = v.x; d[t][3] = v.y;
          } else {
            mma<false>(d[t], a(t)[i], b(t)[sum - i][0], b(t)[sum - i][1]);
          }
        }
}
// ---- sums over the earlier (or later) tokens of a chunk ---------------------------------------------------------------
// They are products over all 16 with zeros in the other places, and zero times a NaN or an infinity is a NaN: a value that is not
// finite would reach tokens that do not depend on it.  In a product it reaches every result of its column (or row), so a look at
// one of them finds it; the product is then formed again a token at a time, with the other tokens' values set to zero, and
// added where the token counts.  (The look costs 0.5 %: (16, 4, 2048, N 48 fp16) forward + backward through autograd 681 -> 684 us;
// with the first turn's operands kept for the second one they were spilled in every chunk, 694.)
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }
// what is kept for token i in a register that holds the tokens k0, k0 + 1
__device__ __forceinline__ uint32_t only_token(int i, int k0) { return i == k0 ? 0x0000ffffu : i == k0 + 1 ? 0xffff0000u : 0u; }
__device__ __forceinline__ uint32_t transposed(uint32_t w) {   // an 8 x 8 tile of pairs across the warp
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(w));
  return r;
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const uint8_t* row) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(row);
  if constexpr (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

constexpr int TABF = 17 * TABW * 2 + 10 * L;                         // floats of one table
constexpr int V_H = 17 * TABW * 2, V_KAPPA = V_H + 2 * L, V_KC = V_H + 4 * L, V_MNEXT = V_H + 6 * L, V_HLOW = V_H + 8 * L;

enum Mode { FORWARD, SWEEP_A, STATES, SWEEP_B, ADJ_STATES };

// Shared memory of a CTA.  Raw rows are in the tensors' types, two chunks of each but of rows that are converted first.
struct Layout {
  int pD, pU, pY, pP;                       // row pitches in bytes
  int b, c, u, y, raw_end, up, yp, tab, part, dpart, red, sig, dd, bytes;
  __host__ __device__ constexpr Layout(int W, int esz, int ysz, int nu, int ny, Mode mode)
      : pD(row_pitch(32 * W * esz)), pU(row_pitch(ROWS * esz)), pY(row_pitch(ROWS * ysz)), pP(row_pitch(ROWS * 2)), b(0), c(0),
        u(0), y(0), raw_end(0), up(0), yp(0), tab(0), part(0), dpart(0), red(0), sig(0), dd(0), bytes(0) {
    const bool back = mode == SWEEP_A || mode == SWEEP_B, dy = back || mode == ADJ_STATES, cross = mode == FORWARD || mode == SWEEP_B;
    int o = 0;
    b = o; o += mode != ADJ_STATES ? 2 * L * pD : 0;
    c = o; o += mode != STATES ? 2 * L * pD : 0;
    u = o; o += mode != ADJ_STATES ? (nu > 1 ? 1 : 2) * L * pU : 0;
    y = o; o += dy ? (ny > 1 ? 1 : 2) * L * pY : 0;
    raw_end = o;
    up = o; o += mode != ADJ_STATES && nu > 1 ? nu * L * pP : 0;   // rows of U and dY as bfloat16 parts
    yp = o; o += dy && ny > 1 ? ny * L * pP : 0;
    tab = o; o += 2 * TABF * 4;                                    // P(j, i); h, P(L,i) h, kc, m behind the token, rest of h
    part = o; o += cross ? W * 8 * 32 * 16 : 0;                    // sums over a warp's columns, by fragment
    dpart = o; o += cross ? W * 4 * 32 * 16 : 0;                   // <c_j, b_i> over a warp's columns, by fragment
    red = o; o += back ? 2 * W * L * 8 : 0;                        // a warp's part of the per-token scalars, of two chunks
    sig = o; o += back ? W * L * 4 : 0;                            // X(i,i), a copy for each warp
    dd = o; o += mode == SWEEP_B ? 2 * L * 16 : 0;                 // X(i,i) conj(d(i,i)) and m behind the token, of two chunks
    bytes = o;
  }
};

__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Rows [0, nb) of cols elements, pitch elements apart in memory, into shared memory.  16-byte pieces where every row starts
// on such a boundary and is a whole number of them, element by element where not.
template <typename T>
__device__ __forceinline__ void stage_rows(uint8_t* dst, int dst_pitch, const T* src, int nb, int cols, int pitch) {
  const int bytes = cols * (int)sizeof(T);
  if (((reinterpret_cast<uintptr_t>(src) | (uintptr_t)bytes | (uintptr_t)(pitch * (int)sizeof(T))) & 15) == 0) {
    const int pieces = bytes >> 4;   // (at most 64, so the reciprocal is exact for the at most 1024 indexes)
    const unsigned inv = 65536u / pieces + 1;
#pragma unroll 1
    for (int i = threadIdx.x; i < nb * pieces; i += blockDim.x) {
      const int r = (int)(((unsigned)i * inv) >> 16), k = i - r * pieces;
      cp_async16(dst + r * dst_pitch + 16 * k, reinterpret_cast<const uint8_t*>(src + (size_t)r * pitch) + 16 * k);
    }
  } else {
#pragma unroll 1
    for (int r = threadIdx.x >> 5; r < nb; r += blockDim.x >> 5)
#pragma unroll 1
      for (int k = threadIdx.x & 31; k < cols; k += 32) reinterpret_cast<T*>(dst + r * dst_pitch)[k] = src[(size_t)r * pitch + k];
  }
}

// columns 2q, 2q + 1 of a raw row as pairs of real and of imaginary parts
template <typename T> __device__ __forceinline__ void raw_complex2(const uint8_t* row, int q, f2& re, f2& im) {
  float2 a, b;
  if constexpr (sizeof(T) == 2) {
    const uint2 w = reinterpret_cast<const uint2*>(row)[q];
    a = unpack_pair<T>(w.x); b = unpack_pair<T>(w.y);
  } else {
    const float4 w = reinterpret_cast<const float4*>(row)[q];
    a = make_float2(w.x, w.y); b = make_float2(w.z, w.w);
  }
  re = mk2(a.x, b.x); im = mk2(a.y, b.y);
}
// column n of two successive raw rows, as pairs over the rows
template <typename T> __device__ __forceinline__ void raw_tokens2(const uint8_t* row, int pitch, int n, f2& re, f2& im) {
  float2 a, b;
  if constexpr (sizeof(T) == 2) {
    a = unpack_pair<T>(reinterpret_cast<const uint32_t*>(row)[n]);
    b = unpack_pair<T>(reinterpret_cast<const uint32_t*>(row + pitch)[n]);
  } else {
    a = reinterpret_cast<const float2*>(row)[n];
    b = reinterpret_cast<const float2*>(row + pitch)[n];
  }
  re = mk2(a.x, b.x); im = mk2(a.y, b.y);
}
template <typename T> __device__ __forceinline__ void raw_quad(const uint8_t* row, int q, f2 (&v)[2]) {   // elements 4q .. 4q + 3
  if constexpr (sizeof(T) == 2) {
    const uint2 w = reinterpret_cast<const uint2*>(row)[q];
    const float2 a = unpack_pair<T>(w.x), b = unpack_pair<T>(w.y);
    v[0] = mk2(a.x, a.y); v[1] = mk2(b.x, b.y);
  } else {
    const float4 w = reinterpret_cast<const float4*>(row)[q];
    v[0] = mk2(w.x, w.y); v[1] = mk2(w.z, w.w);
  }
}
__device__ __forceinline__ float hsum(f2 v) { const float2 q = un2(v); return q.x + q.y; }
__device__ __forceinline__ f2 neg2(f2 v) { return mul2(v, dup2(-1.f)); }
// (ar + i ai)(br + i bi) and its conjugated form conj(a) b, elementwise on pairs
__device__ __forceinline__ void cmul2(f2 ar, f2 ai, f2 br, f2 bi, f2& re, f2& im) {
  re = fma2(neg2(ai), bi, mul2(ar, br)); im = fma2(ai, br, mul2(ar, bi));
}
__device__ __forceinline__ void cmul2_conj_a(f2 ar, f2 ai, f2 br, f2 bi, f2& re, f2& im) {
  re = fma2(ai, bi, mul2(ar, br)); im = fma2(neg2(ai), br, mul2(ar, bi));
}
// the latter added to re, im
__device__ __forceinline__ void cmac2_conj_a(f2 ar, f2 ai, f2 br, f2 bi, f2& re, f2& im) {
  re = fma2(ar, br, fma2(ai, bi, re)); im = fma2(ar, bi, fma2(neg2(ai), br, im));
}
__device__ __forceinline__ cf load_cf(const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return {v.x, v.y}; }
__device__ __forceinline__ void store_cf(float* p, cf v) { *reinterpret_cast<float2*>(p) = make_float2(v.re, v.im); }
// two successive complex numbers ``step`` floats apart as pairs
__device__ __forceinline__ void load_cf2(const float* p, int step, f2& re, f2& im) {
  const cf a = load_cf(p), b = load_cf(p + step);
  re = mk2(a.re, b.re); im = mk2(a.im, b.im);
}
template <typename T> __device__ __forceinline__ cf load_c(const T* base, size_t cidx) {
  return {to_f32(base[2 * cidx]), to_f32(base[2 * cidx + 1])};
}
// two neighbouring elements of an array that may start anywhere; the second only if there is one
template <typename T> __device__ __forceinline__ void store_two(T* dst, bool vec, float a, float b, bool second) {
  if (vec && second) {
    if constexpr (sizeof(T) == 2) *reinterpret_cast<uint32_t*>(dst) = pack_pair<T>(a, b);
    else *reinterpret_cast<float2*>(dst) = make_float2(a, b);
  } else {
    dst[0] = from_f32<T>(a);
    if (second) dst[1] = from_f32<T>(b);
  }
}
__device__ __forceinline__ void put(float* dst, float v, bool add) {
  if (add) atomicAdd(dst, v); else *dst = v;
}

// Where a thread sits in its warp's 16 columns x 64 rows of the state, which are the accumulators of 16 x 8 products: 16
// rows of 8 real and 8 imaginary parts.  Lane (g, q) holds column 8 grp + g of the warp's, rows 8 pt + 2q, + 1 of P.
struct Place {
  int lane, w, g, q;
  __device__ __forceinline__ Place() {
    lane = threadIdx.x & 31; w = threadIdx.x >> 5;
    g = lane >> 2; q = lane & 3;
  }
};
struct Tile { f2 re[2][8], im[2][8]; };

// f(grp, pt, re pair, im pair) for the tile of src (P, 2N), zeros outside.  VEC: src is aligned to a complex number.
template <bool VEC, typename F>
__device__ __forceinline__ void read_tile(const float* src, const Place& o, int row0, int P, int N, F f) {
#pragma unroll
  for (int grp = 0; grp < 2; ++grp)
#pragma unroll
    for (int pt = 0; pt < 8; ++pt) {
      const int n = 16 * o.w + 8 * grp + o.g;
      cf v[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = row0 + 8 * pt + 2 * o.q + e;
        const float* x = src + (size_t)row * 2 * N + 2 * n;
        if (row < P && n < N) v[e] = VEC ? load_cf(x) : cf{x[0], x[1]};
      }
      f(grp, pt, mk2(v[0].re, v[1].re), mk2(v[0].im, v[1].im));
    }
}
template <bool VEC>
__device__ __forceinline__ void store_tile(const Tile& z, float* dst, const Place& o, int row0, int P, int N) {
#pragma unroll
  for (int grp = 0; grp < 2; ++grp)
#pragma unroll
    for (int pt = 0; pt < 8; ++pt) {
      const int n = 16 * o.w + 8 * grp + o.g;
      const float2 re = un2(z.re[grp][pt]), im = un2(z.im[grp][pt]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = row0 + 8 * pt + 2 * o.q + e;
        float* x = dst + (size_t)row * 2 * N + 2 * n;
        if (row < P && n < N) {
          const cf v = {e ? re.y : re.x, e ? im.y : im.x};
          if (VEC) store_cf(x, v);
          else { x[0] = v.re; x[1] = v.im; }
        }
      }
    }
}
// z = m z (CONJ: conj(m) z)
template <bool CONJ>
__device__ __forceinline__ void scale_tile(Tile& z, cf m) {
  const f2 r2 = dup2(m.re), i2 = dup2(CONJ ? -m.im : m.im), n2 = dup2(CONJ ? m.im : -m.im);
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const f2 a = z.re[r][i], b = z.im[r][i];
      z.re[r][i] = fma2(n2, b, mul2(r2, a));
      z.im[r][i] = fma2(i2, a, mul2(r2, b));
    }
}
// Product of the transitions [t0, t1) (1 past the end of the sequence), by one warp, to dst.
__device__ __forceinline__ void transition_product(const float* Mb, int t0, int t1, int T, float* dst) {
  const int lane = threadIdx.x & 31;
  double re = 1.0, im = 0.0;
#pragma unroll 1
  for (int t = t0 + lane; t < t1; t += 32) {
    if (t >= T) continue;
    const double mr = Mb[2 * t], mi = Mb[2 * t + 1], r = re * mr - im * mi;
    im = re * mi + im * mr; re = r;
  }
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    const double orr = __shfl_xor_sync(0xffffffffu, re, o), oi = __shfl_xor_sync(0xffffffffu, im, o);
    const double r = re * orr - im * oi;
    im = re * oi + im * orr; re = r;
  }
  if (lane == 0) { dst[0] = (float)re; dst[1] = (float)im; }
}

// The products of one chunk, by one warp.  Lane l stands for the source token i = l - 1 (l = 0: the chunk's start state):
// tab[j][l] = P(j, i), then per source h, P(nb, i) h, kc, the transition behind it and what float32 leaves of h.  In
// float64, rounded once: an error of a product is common to all rows and columns of the state, so the sums over them do not
// average it out as they do the roundings of a walk token by token (dU and dB came 10 to 15 % further from float64 with
// float32 products).
struct ChainIn { float2 m, kp, kc; };
__device__ __forceinline__ ChainIn load_chain(const float* M, const float* K, int t0, int T, int lane) {
  ChainIn in{make_float2(1.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  const int t = t0 + lane;
  if (lane <= L) {
    if (t < T) {
      in.m = *reinterpret_cast<const float2*>(M + 2 * (size_t)t);
      in.kp = *reinterpret_cast<const float2*>(K + 4 * (size_t)t);
    }
    if (lane > 0 && t - 1 < T) in.kc = *reinterpret_cast<const float2*>(K + 4 * (size_t)(t - 1) + 2);
  }
  return in;
}
struct cd { double re, im; };
__device__ __forceinline__ cd cmul(cd a, cd b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cf rounded(cd a) { return {(float)a.re, (float)a.im}; }
__device__ __forceinline__ cd coefficient(const ChainIn& in) {   // h
  const cd v = cmul(cd{in.m.x, in.m.y}, cd{in.kc.x, in.kc.y});
  return {v.re + in.kp.x, v.im + in.kp.y};
}
// The whole table.  The chains of the first nine tokens and of the others run side by side in different lanes, and meet in
// P(j, i) = P(9, i) P(j, 8): this warp's chain is what the others of its CTA wait for.
__device__ __forceinline__ void chain(float* tab, const ChainIn& in, int nb, int lane) {
  const bool hi = lane >= 9;
  cd p = {1.0, 0.0}, end = {1.0, 0.0}, q[7];
  if (lane == 0 || lane == 9) store_cf(tab + 2 * (lane * TABW + lane), {1.f, 0.f});
#pragma unroll
  for (int s = 1; s <= 9; ++s) {
    const int j = hi ? 9 + s : s;
    const cd m = {__shfl_sync(0xffffffffu, in.m.x, j & 31), __shfl_sync(0xffffffffu, in.m.y, j & 31)};
    if (lane < j && j <= L) p = cmul(p, m);
    if (lane <= j && j <= L && lane <= L) store_cf(tab + 2 * (j * TABW + lane), rounded(p));
    if (j == nb) end = p;
    if (s <= 7) q[s - 1] = {__shfl_sync(0xffffffffu, p.re, 9), __shfl_sync(0xffffffffu, p.im, 9)};
  }
#pragma unroll
  for (int s = 1; s <= 7; ++s) {
    const cd v = cmul(p, q[s - 1]);
    if (!hi) {
      store_cf(tab + 2 * ((9 + s) * TABW + lane), rounded(v));
      if (9 + s == nb) end = v;
    }
  }
  if (lane >= 1 && lane <= L) {
    const int i = lane - 1;
    const cd h = coefficient(in);
    const cf hf = rounded(h);
    store_cf(tab + V_H + 2 * i, hf);
    store_cf(tab + V_HLOW + 2 * i, {(float)(h.re - hf.re), (float)(h.im - hf.im)});
    store_cf(tab + V_KAPPA + 2 * i, rounded(cmul(end, h)));
    store_cf(tab + V_KC + 2 * i, {in.kc.x, in.kc.y});
    store_cf(tab + V_MNEXT + 2 * i, {in.m.x, in.m.y});
  }
}
// What the pre-passes need of it: forward in time P(L, i) h_i (a chunk that is shorter ends in transitions of 1) and a_nb, the
// adjoint's a_j; products over all later or all earlier lanes.
template <bool ADJ>
__device__ __forceinline__ void chain_ends(float* tab, const ChainIn& in, int nb, int lane) {
  const bool own = lane >= 1 && lane <= L;
  cd p = {own ? in.m.x : 1.0, own ? in.m.y : 0.0};
#pragma unroll
  for (int o = 1; o <= L; o <<= 1) {
    const cd v = {ADJ ? __shfl_up_sync(0xffffffffu, p.re, o) : __shfl_down_sync(0xffffffffu, p.re, o),
                  ADJ ? __shfl_up_sync(0xffffffffu, p.im, o) : __shfl_down_sync(0xffffffffu, p.im, o)};
    if (ADJ ? lane >= o : lane + o < 32) p = cmul(p, v);
  }
  if (ADJ) {
    if (lane <= L) store_cf(tab + 2 * lane * TABW, rounded(p));
  } else {
    const cd end = {__shfl_down_sync(0xffffffffu, p.re, 1), __shfl_down_sync(0xffffffffu, p.im, 1)};   // over the lanes behind this one
    if (own) store_cf(tab + V_KAPPA + 2 * (lane - 1), rounded(cmul(end, coefficient(in))));
    if (lane == 0) store_cf(tab + 2 * nb * TABW, rounded(end));
  }
}

// One walk of one segment.  FORWARD: Y and the final state.  SWEEP_A / SWEEP_B: the two sweeps of the backward.  STATES /
// ADJ_STATES: only where the segment ends, from zero.
template <typename TIn, typename TY, Mode MODE>
__device__ __forceinline__ void walk(const SweepParams& p, int pt0, int seg, uint8_t* smem) {
  constexpr bool REV = MODE == SWEEP_B || MODE == ADJ_STATES, BACK = MODE == SWEEP_A || MODE == SWEEP_B;
  constexpr bool ONLY_STATES = MODE == STATES || MODE == ADJ_STATES;
  constexpr bool USE_B = MODE != ADJ_STATES, USE_C = MODE != STATES, USE_DY = BACK || MODE == ADJ_STATES, USE_U = USE_B;
  constexpr int NI = Parts<TIn>::N, NY = Parts<TY>::N;
  const int W = p.W, N = p.N, P = p.P, T = p.T, D = 2 * N, NT = 32 * W;
  const Layout lay(W, sizeof(TIn), sizeof(TY), NI, NY, MODE);
  const Place o;
  const int tid = threadIdx.x;
  const int h = blockIdx.x, b = blockIdx.y, bh = b * p.heads + h, bg = b * p.groups + h / (p.heads / p.groups);
  const int row0 = pt0 * ROWS, prows = min(ROWS, P - row0);
  const TIn* U = reinterpret_cast<const TIn*>(p.U) + (size_t)bh * T * P + row0;
  const TIn* B = reinterpret_cast<const TIn*>(p.B) + (size_t)bg * T * D;
  const TIn* C = reinterpret_cast<const TIn*>(p.C) + (size_t)bg * T * D;
  const TY* dY = p.dY ? reinterpret_cast<const TY*>(p.dY) + (size_t)bh * T * P + row0 : nullptr;
  const float* M = p.M + (size_t)bh * T * 2;
  const float* K = p.K + (size_t)bh * T * 4;
  const int t_lo = seg * p.seg_len, t_hi = min(T, t_lo + p.seg_len), nchunks = (t_hi - t_lo + L - 1) / L;
  float* tabs = reinterpret_cast<float*>(smem + lay.tab);
  float4* part = reinterpret_cast<float4*>(smem + lay.part);
  float4* dpart = reinterpret_cast<float4*>(smem + lay.dpart);
  float* red = reinterpret_cast<float*>(smem + lay.red);
  float* sig = reinterpret_cast<float*>(smem + lay.sig) + o.w * L;
  float4* dd = reinterpret_cast<float4*>(smem + lay.dd);
  auto first_of = [&](int c) { return t_lo + L * (REV ? nchunks - 1 - c : c); };   // first token of the walk's chunk c
  auto raw = [&](int base, int pitch, int c, int j) { return smem + base + ((c & 1) * L + j) * pitch; };

  auto raw_u = [&](int c) { return smem + lay.u + (NI > 1 ? 0 : (c & 1) * L * lay.pU); };
  auto raw_y = [&](int c) { return smem + lay.y + (NY > 1 ? 0 : (c & 1) * L * lay.pY); };
  // tensors whose rows are converted are staged behind that, the others at the start of the chunk before
  auto stage = [&](int c, bool converted) {
    const int t0 = first_of(c), nb = min(L, t_hi - t0);
    if (USE_U && converted == (NI > 1)) stage_rows<TIn>(raw_u(c), lay.pU, U + (size_t)t0 * P, nb, prows, P);
    if (USE_DY && dY && converted == (NY > 1)) stage_rows<TY>(raw_y(c), lay.pY, dY + (size_t)t0 * P, nb, prows, P);
    if (converted) return;
    if (USE_B) stage_rows<TIn>(raw(lay.b, lay.pD, c, 0), lay.pD, B + (size_t)t0 * D, nb, D, D);
    if (USE_C) stage_rows<TIn>(raw(lay.c, lay.pD, c, 0), lay.pD, C + (size_t)t0 * D, nb, D, D);
  };
  // rows of U or dY as bfloat16 parts; bfloat16 rows are their own
  auto convert = [&](auto type, const uint8_t* rows, int pitch, int parts) {
    using X = decltype(type);
    constexpr int NP = Parts<X>::N;
#pragma unroll 1
    for (int i = tid; i < L * ROWS / 4; i += NT) {
      f2 v[2];
      raw_quad<X>(rows + (i >> 4) * pitch, i & 15, v);
      uint32_t w0[NP], w1[NP];
      split<NP>(v[0], w0); split<NP>(v[1], w1);
#pragma unroll
      for (int k = 0; k < NP; ++k)
        *reinterpret_cast<uint2*>(smem + parts + (k * L + (i >> 4)) * lay.pP + 8 * (i & 15)) = make_uint2(w0[k], w1[k]);
    }
  };
  auto u_rows = [&](int c, int k) -> const uint8_t* { return NI == 1 ? raw_u(c) : smem + lay.up + k * L * lay.pP; };
  auto y_rows = [&](int c, int k) -> const uint8_t* { return NY == 1 ? raw_y(c) : smem + lay.yp + k * L * lay.pP; };
  static_assert(row_pitch(ROWS * 2) == 144, "raw bfloat16 rows and parts have one pitch");
  constexpr int PP = 144;
  const int r_lo = ((o.lane & 7) + 8 * ((o.lane >> 3) & 1)) * PP + 16 * (o.lane >> 4);     // ldmatrix: 16 tokens first, then 16 rows of P
  const int r_hi = ((o.lane & 7) + 8 * (o.lane >> 4)) * PP + 16 * ((o.lane >> 3) & 1);     // and the other way round

  // Columns beyond N and rows beyond P stay zero for good.  (So do the tokens that a ragged chunk has not in a walk backwards,
  // which begins with it; forward in time such tokens have h = 0, and their results are not stored.)
#pragma unroll 1
  for (int i = tid; i < lay.raw_end / 16; i += NT) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  stage(0, false);
  stage(0, true);
  auto products_of = [&](int c, const ChainIn& in) {   // one warp
    float* tab = tabs + (c & 1) * TABF;
    const int nb = min(L, t_hi - first_of(c));
    if constexpr (ONLY_STATES) chain_ends<REV>(tab, in, nb, o.lane);
    else chain(tab, in, nb, o.lane);
  };
  if (o.w == 0) products_of(0, load_chain(M, K, first_of(0), T, o.lane));

  // ---- start state -------------------------------------------------------------------------------------------------
  Tile z;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int i = 0; i < 8; ++i) z.re[r][i] = z.im[r][i] = 0ull;
  if (!ONLY_STATES) {
    auto take = [&](int r, int i, f2 re, f2 im) { z.re[r][i] = re; z.im[r][i] = im; };
    if (p.nseg > 1) {   // combined by the launch before
      read_tile<true>((REV ? p.gloc : p.zloc) + ((size_t)seg * p.batch * p.heads + bh) * P * D, o, row0, P, N, take);
    } else if (REV) {
      if (p.dfinal) read_tile<false>(p.dfinal + (size_t)bh * P * D, o, row0, P, N, take);
    } else {
      if (p.z0) {
        read_tile<false>(p.z0 + (size_t)bh * P * D, o, row0, P, N, take);
        scale_tile<false>(z, load_cf(M));
      }
      if (p.Bprev) {   // the prev-tap of the first token
        const TIn* Bp = reinterpret_cast<const TIn*>(p.Bprev) + (size_t)bg * D;
        const TIn* Up = reinterpret_cast<const TIn*>(p.Uprev) + (size_t)bh * P + row0;
        const cf kp = load_cf(K);
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) {
          const int n = 16 * o.w + 8 * grp + o.g;
          const cf x = n < N ? cmul(kp, load_c(Bp, n)) : cf{0.f, 0.f};
#pragma unroll
          for (int pt = 0; pt < 8; ++pt) {
            const int r = 8 * pt + 2 * o.q;
            const f2 u = mk2(r < prows ? to_f32(Up[r]) : 0.f, r + 1 < prows ? to_f32(Up[r + 1]) : 0.f);
            z.re[grp][pt] = fma2(u, dup2(x.re), z.re[grp][pt]);
            z.im[grp][pt] = fma2(u, dup2(x.im), z.im[grp][pt]);
          }
        }
      }
    }
  } else if (pt0 == 0 && o.w == W - 1) {
    transition_product(M, t_lo + 1, t_hi + 1, T, (REV ? p.gprod : p.zprod) + 2 * ((size_t)seg * p.batch * p.heads + bh));
  }

  // per-token scalars of chunk c from the warps' parts; warp W - 1, after the barrier that follows the chunk
  auto finish_scalars = [&](int c) {
    const int t0 = first_of(c), nb = min(L, t_hi - t0), j = o.lane;
    if (o.w != W - 1 || j >= nb) return;
    float re = 0.f, im = 0.f;
#pragma unroll 1
    for (int k = 0; k < W; ++k) { const cf v = load_cf(red + 2 * (((c & 1) * W + k) * L + j)); re += v.re; im += v.im; }
    const size_t t = (size_t)bh * T + t0 + j;
    const bool add = p.ptiles > 1;
    if (MODE == SWEEP_A) { put(p.sterm + 2 * t, re, add); put(p.sterm + 2 * t + 1, im, add); }
    if (MODE == SWEEP_B) {
      float* dkp = t0 + j + 1 < T ? p.dK + 4 * (t + 1) : p.dM + 2 * t;   // dkp of the next token; the last one's for finish_dm
      put(dkp, re, add); put(dkp + 1, im, add);
      const float4 sd = dd[(c & 1) * L + j];
      const cf g = cmul_conj_a({sd.z, sd.w}, {re, im});
      put(p.dK + 4 * t + 2, g.re + sd.x, add); put(p.dK + 4 * t + 3, g.im + sd.y, add);
    }
  };

  for (int c = 0; c < nchunks; ++c) {
    const int t0 = first_of(c), nb = min(L, t_hi - t0);
    const float* tab = tabs + (c & 1) * TABF;
    cp_async_wait();
    __syncthreads();
    if (BACK && c > 0) finish_scalars(c - 1);
    ChainIn next{};
    if (c + 1 < nchunks) {
      stage(c + 1, false);
      if (o.w == 0) next = load_chain(M, K, first_of(c + 1), T, o.lane);
    }
    if ((USE_U && NI > 1) || (USE_DY && NY > 1)) {
      if (USE_U && NI > 1) convert(TIn{}, raw_u(c), lay.pU, lay.up);
      if (USE_DY && NY > 1) convert(TY{}, raw_y(c), lay.pY, lay.yp);
      __syncthreads();
      if (c + 1 < nchunks) stage(c + 1, true);
    }
    // column 8 grp + g of the warp's at the tokens 8 tt + 2q, + 1, as pairs over the tokens
    auto tokens_of = [&](int base, int grp, int tt, f2& re, f2& im) {
      raw_tokens2<TIn>(raw(base, lay.pD, c, 8 * tt + 2 * o.q), lay.pD, 16 * o.w + 8 * grp + o.g, re, im);
    };
    // columns 8 grp + 2q, + 1 at token 8 tt + g, as pairs over the columns
    auto columns_of = [&](int base, int grp, int tt, f2& re, f2& im) {
      raw_complex2<TIn>(raw(base, lay.pD, c, 8 * tt + o.g), 8 * o.w + 4 * grp + o.q, re, im);
    };

    // ---- <c_j, b_i> over the warp's columns: rows j (SWEEP_B: i), columns i (j) ---------------------------------------
    if (MODE == FORWARD || MODE == SWEEP_B) {
      f2 re[2][2], im[2][2];   // [column tile][row half]
#pragma unroll
      for (int k = 0; k < 4; ++k) re[k >> 1][k & 1] = im[k >> 1][k & 1] = 0ull;
#pragma unroll
      for (int grp = 0; grp < 2; ++grp) {
        uint32_t a[NI][4];
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          f2 r, i;
          uint32_t wr[NI], wi[NI];
          columns_of(MODE == FORWARD ? lay.c : lay.b, grp, tt, r, i);
          split<NI>(r, wr); split<NI>(i, wi);
#pragma unroll
          for (int k = 0; k < NI; ++k) { a[k][tt] = wr[k]; a[k][2 + tt] = wi[k]; }
        }
        uint32_t x[4][NI][2];   // [column tile: re, im]
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          f2 r, i;
          uint32_t wr[NI], wi[NI];
          columns_of(MODE == FORWARD ? lay.b : lay.c, grp, tt, r, i);
          split<NI>(r, wr); split<NI>(i, wi);
#pragma unroll
          for (int k = 0; k < NI; ++k) {
            x[2 * tt][k][0] = wr[k]; x[2 * tt][k][1] = wi[k];
            // Im <c, b> = c_re b_im - c_im b_re
            x[2 * tt + 1][k][0] = MODE == FORWARD ? wi[k] : wi[k] ^ 0x80008000u;
            x[2 * tt + 1][k][1] = MODE == FORWARD ? wr[k] ^ 0x80008000u : wr[k];
          }
        }
        float d[4][4];
        products<4, NI, NI>(d, [&](int) { return &a[0]; }, [&](int t) { return &x[t][0]; });
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          re[tt][0] = add2(re[tt][0], mk2(d[2 * tt][0], d[2 * tt][1])); re[tt][1] = add2(re[tt][1], mk2(d[2 * tt][2], d[2 * tt][3]));
          im[tt][0] = add2(im[tt][0], mk2(d[2 * tt + 1][0], d[2 * tt + 1][1]));
          im[tt][1] = add2(im[tt][1], mk2(d[2 * tt + 1][2], d[2 * tt + 1][3]));
        }
      }
#pragma unroll
      for (int tt = 0; tt < 2; ++tt) {
        const float2 r0 = un2(re[tt][0]), r1 = un2(re[tt][1]), i0 = un2(im[tt][0]), i1 = un2(im[tt][1]);
        dpart[(o.w * 4 + 2 * tt) * 32 + o.lane] = make_float4(r0.x, r0.y, r1.x, r1.y);
        dpart[(o.w * 4 + 2 * tt + 1) * 32 + o.lane] = make_float4(i0.x, i0.y, i1.x, i1.y);
      }
    }

    // ---- products with the state at the chunk's start -----------------------------------------------------------------
    f2 hre[2][2], him[2][2];   // SWEEP_A, SWEEP_B: sum over the rows of P of dy_j (u_i) times the state, [grp][token tile]
    if (!ONLY_STATES) {
      constexpr bool CROSS = MODE != SWEEP_A;
      uint32_t op[2][3][4];    // FORWARD: conj(a_j) c_j, SWEEP_B: P(L,i) h_i b_i; rows tokens
      if (CROSS) {
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          const cf s = load_cf(MODE == FORWARD ? tab + 2 * (8 * tt + o.g) * TABW : tab + V_KAPPA + 2 * (8 * tt + o.g));
#pragma unroll
          for (int grp = 0; grp < 2; ++grp) {
            f2 r, i, xr, xi;
            uint32_t wr[3], wi[3];
            columns_of(MODE == FORWARD ? lay.c : lay.b, grp, tt, r, i);
            if (MODE == FORWARD) cmul2_conj_a(dup2(s.re), dup2(s.im), r, i, xr, xi);
            else cmul2(dup2(s.re), dup2(s.im), r, i, xr, xi);
            split<3>(xr, wr); split<3>(xi, wi);
#pragma unroll
            for (int k = 0; k < 3; ++k) { op[grp][k][tt] = wr[k]; op[grp][k][2 + tt] = wi[k]; }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) hre[k >> 1][k & 1] = him[k >> 1][k & 1] = 0ull;
#pragma unroll
      for (int s = 0; s < 4; ++s) {   // 16 rows of P at a time
        constexpr int NR = MODE == SWEEP_A ? NY : NI;
        uint32_t rows[2][NR][2];      // [token tile]
        if (BACK)
#pragma unroll
          for (int k = 0; k < NR; ++k) {
            uint32_t r[4];
            ldmatrix4<false>(r, (MODE == SWEEP_A ? y_rows(c, k) : u_rows(c, k)) + r_hi + 32 * s);
            rows[0][k][0] = r[0]; rows[0][k][1] = r[1]; rows[1][k][0] = r[2]; rows[1][k][1] = r[3];
          }
        f2 y0[2], y1[2];              // FORWARD, SWEEP_B: [pt]: tokens g and 8 + g
        uint32_t a[2][3][4];
#pragma unroll
        for (int grp = 0; grp < 2; ++grp)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            uint32_t wr[3], wi[3];
            split<3>(z.re[grp][2 * s + k], wr); split<3>(z.im[grp][2 * s + k], wi);
#pragma unroll
            for (int x = 0; x < 3; ++x) { a[grp][x][2 * k] = wr[x]; a[grp][x][2 * k + 1] = wi[x]; }
          }
        if (BACK) {
          float d[4][4];   // [grp, token tile]
          products<4, 3, NR>(d, [&](int t) { return &a[t >> 1][0]; }, [&](int t) { return &rows[t & 1][0]; });
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            hre[t >> 1][t & 1] = add2(hre[t >> 1][t & 1], mk2(d[t][0], d[t][1]));
            him[t >> 1][t & 1] = add2(him[t >> 1][t & 1], mk2(d[t][2], d[t][3]));
          }
        }
        if (CROSS) {
          uint32_t x[4][3][2];   // [grp, pt]
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 3; ++e) {
              x[t][e][0] = transposed(a[t >> 1][e][2 * (t & 1)]); x[t][e][1] = transposed(a[t >> 1][e][2 * (t & 1) + 1]);
            }
          float d[4][4];
          products<4, 3, 3, true>(d, [&](int t) { return &op[t >> 1][0]; }, [&](int t) { return &x[t][0]; });
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            y0[k] = add2(mk2(d[k][0], d[k][1]), mk2(d[2 + k][0], d[2 + k][1]));
            y1[k] = add2(mk2(d[k][2], d[k][3]), mk2(d[2 + k][2], d[2 + k][3]));
          }
        }
        if (CROSS)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float2 v0 = un2(y0[k]), v1 = un2(y1[k]);
            part[(o.w * 8 + 2 * s + k) * 32 + o.lane] = make_float4(v0.x, v0.y, v1.x, v1.y);
          }
      }
    }

    // ---- SWEEP_A, SWEEP_B: the chunk's own part, dC / dB and the scalars -----------------------------------------------
    if (BACK) {
      // X(j,i) = <dy_j, u_i>: rows j, columns i in SWEEP_A, the other way round in SWEEP_B
      constexpr int NA = MODE == SWEEP_A ? NY : NI, NB = MODE == SWEEP_A ? NI : NY;
      f2 x[2][2];   // [column tile][row half]
      x[0][0] = x[0][1] = x[1][0] = x[1][1] = 0ull;
#pragma unroll
      for (int s = 0; s < 4; s += 2) {
        uint32_t a[2][NA][4], r[4][NB][2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int k = 0; k < NA; ++k) ldmatrix4<false>(a[e][k], (MODE == SWEEP_A ? y_rows(c, k) : u_rows(c, k)) + r_lo + 32 * (s + e));
#pragma unroll
          for (int k = 0; k < NB; ++k) {
            uint32_t v[4];
            ldmatrix4<false>(v, (MODE == SWEEP_A ? u_rows(c, k) : y_rows(c, k)) + r_hi + 32 * (s + e));
            r[2 * e][k][0] = v[0]; r[2 * e][k][1] = v[1]; r[2 * e + 1][k][0] = v[2]; r[2 * e + 1][k][1] = v[3];
          }
        }
        float d[4][4];   // [rows of P, column tile]
        products<4, NA, NB, true>(d, [&](int t) { return &a[t >> 1][0]; }, [&](int t) { return &r[t][0]; });
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          x[t][0] = add2(x[t][0], add2(mk2(d[t][0], d[t][1]), mk2(d[2 + t][0], d[2 + t][1])));
          x[t][1] = add2(x[t][1], add2(mk2(d[t][2], d[t][3]), mk2(d[2 + t][2], d[2 + t][3])));
        }
      }
      if (o.q == (o.g >> 1)) {   // the diagonal
        const float2 v0 = un2(x[0][0]), v1 = un2(x[1][1]);
        sig[o.g] = (o.g & 1) ? v0.y : v0.x;
        sig[8 + o.g] = (o.g & 1) ? v1.y : v1.x;
      }
      __syncwarp();
      // times the coefficients, below the diagonal: A  P(j,i) h_i,  B  conj(P(j,i)); columns of the product below
      uint32_t x3[4][3][2];   // [real, imaginary; token tile]
#pragma unroll
      for (int tt = 0; tt < 2; ++tt)
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int own = 8 * tt + o.g, src = 8 * it + 2 * o.q;   // A: j = own, i = src; B: i = own, j = src
          f2 pr, pi, gr, gi;
          if (MODE == SWEEP_A) {
            f2 hr, hi;
            load_cf2(tab + 2 * (own * TABW + src + 1), 2, pr, pi);
            load_cf2(tab + V_H + 2 * src, 2, hr, hi);
            cmul2(pr, pi, hr, hi, gr, gi);
          } else {
            load_cf2(tab + 2 * (src * TABW + own + 1), 2 * TABW, gr, pi);
            gi = neg2(pi);
          }
          const float2 vr = un2(mul2(x[it][tt], gr)), vi = un2(mul2(x[it][tt], gi));
          const bool m0 = MODE == SWEEP_A ? src < own : src > own, m1 = MODE == SWEEP_A ? src + 1 < own : src + 1 > own;
          uint32_t wr[3], wi[3];
          split<3>(mk2(m0 ? vr.x : 0.f, m1 ? vr.y : 0.f), wr);
          split<3>(mk2(m0 ? vi.x : 0.f, m1 ? vi.y : 0.f), wi);
#pragma unroll
          for (int k = 0; k < 3; ++k) { x3[tt][k][it] = wr[k]; x3[2 + tt][k][it] = wi[k]; }
        }
      const int other = MODE == SWEEP_A ? lay.b : lay.c, self = MODE == SWEEP_A ? lay.c : lay.b;
      f2 sre[2], sim[2];   // <c_j, .>, <b_i, .> over the lane's columns, [token tile]
      sre[0] = sre[1] = sim[0] = sim[1] = 0ull;
#pragma unroll
      for (int grp = 0; grp < 2; ++grp) {
        uint32_t a[2][NI][4];   // (re | im) and (-im | re)
        f2 ore[2], oim[2];
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          uint32_t wr[NI], wi[NI];
          tokens_of(other, grp, tt, ore[tt], oim[tt]);
          split<NI>(ore[tt], wr); split<NI>(oim[tt], wi);
#pragma unroll
          for (int k = 0; k < NI; ++k) {
            a[0][k][2 * tt] = wr[k]; a[0][k][2 * tt + 1] = wi[k];
            a[1][k][2 * tt] = wi[k] ^ 0x80008000u; a[1][k][2 * tt + 1] = wr[k];
          }
        }
        float d[4][4];   // [times the real, the imaginary factors; token tile]
        products<4, NI, 3>(d, [&](int t) { return &a[t >> 1][0]; }, [&](int t) { return &x3[t][0]; });
        if (__any_sync(0xffffffffu, not_finite(d[0][0] + d[0][2]))) {
#pragma unroll
          for (int t = 0; t < 4; ++t) d[t][0] = d[t][1] = d[t][2] = d[t][3] = 0.f;
#pragma unroll 1
          for (int i = 0; i < L; ++i) {
            f2 re, im;   // (read again: registers for the operands of both turns would be spilled in the one that runs)
            uint32_t wr[NI], wi[NI];
            tokens_of(other, grp, i >> 3, re, im);
            split<NI>(re, wr); split<NI>(im, wi);
            const uint32_t lo = only_token(i, 2 * o.q), hi = only_token(i, 8 + 2 * o.q);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              uint32_t one[NI][4];
#pragma unroll
              for (int k = 0; k < NI; ++k) {
                const uint32_t x = t < 2 ? wr[k] : wi[k] ^ 0x80008000u, y = t < 2 ? wi[k] : wr[k];
                one[k][0] = x & lo; one[k][1] = y & lo; one[k][2] = x & hi; one[k][3] = y & hi;
              }
              float e[1][4];
              products<1, NI, 3>(e, [&](int) { return &one[0]; }, [&](int) { return &x3[t][0]; });
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                const int own = 8 * (t & 1) + 2 * o.q + (r & 1);
                if (MODE == SWEEP_A ? i < own : i > own) d[t][r] += e[0][r];
              }
            }
          }
        }
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          const int t = 8 * tt + 2 * o.q;
          f2 er, ei, vr, vi, nr, ni;
          f2 pr = add2(mk2(d[tt][0], d[tt][1]), mk2(d[2 + tt][0], d[2 + tt][1]));
          f2 pi = add2(mk2(d[tt][2], d[tt][3]), mk2(d[2 + tt][2], d[2 + tt][3]));
          if (MODE == SWEEP_A) {   // a_j times the sum
            load_cf2(tab + 2 * t * TABW, 2 * TABW, er, ei);
            cmul2(er, ei, hre[grp][tt], him[grp][tt], vr, vi);
          } else {                 // conj(P(L,i)) times the sum
            load_cf2(tab + 2 * (nb * TABW + t + 1), 2, er, ei);
            cmul2_conj_a(er, ei, hre[grp][tt], him[grp][tt], vr, vi);
          }
          vr = add2(vr, pr); vi = add2(vi, pi);
          f2 sr, si, kr, ki;
          tokens_of(self, grp, tt, sr, si);
          // A: <.., c>: c conj(v); B: conj(b) v
          sre[tt] = fma2(si, vi, fma2(sr, vr, sre[tt]));
          sim[tt] = MODE == SWEEP_A ? fma2(neg2(sr), vi, fma2(si, vr, sim[tt])) : fma2(neg2(si), vr, fma2(sr, vi, sim[tt]));
          load_cf2(tab + V_KC + 2 * t, 2, kr, ki);
          const f2 sg = *reinterpret_cast<const f2*>(sig + t);
          if (MODE == SWEEP_A) {   // + X(j,j) kc_j b_j
            cmul2(mul2(sg, kr), mul2(sg, ki), ore[tt], oim[tt], nr, ni);
            nr = add2(nr, vr); ni = add2(ni, vi);
          } else {                 // conj(h_i) D_i + X(i,i) conj(kc_i) c_i
            f2 hr, hi;
            load_cf2(tab + V_HLOW + 2 * t, 2, hr, hi);
            cmul2_conj_a(hr, hi, vr, vi, nr, ni);
            cmac2_conj_a(mul2(sg, kr), mul2(sg, ki), ore[tt], oim[tt], nr, ni);
            load_cf2(tab + V_H + 2 * t, 2, hr, hi);
            cmac2_conj_a(hr, hi, vr, vi, nr, ni);
          }
          const float2 o_re = un2(nr), o_im = un2(ni);
          const int n = 16 * o.w + 8 * grp + o.g;
#pragma unroll
          for (int e1 = 0; e1 < 2; ++e1) {
            if (n >= N || t + e1 >= nb) continue;
            const float v_re = e1 ? o_re.y : o_re.x, v_im = e1 ? o_im.y : o_im.x;
            if (p.spread) {
              float* dst = (MODE == SWEEP_A ? p.dC_head : p.dB_head) + ((size_t)bh * T + t0 + t + e1) * D + 2 * n;
              put(dst, v_re, p.ptiles > 1); put(dst + 1, v_im, p.ptiles > 1);
            } else {
              TIn* dst = reinterpret_cast<TIn*>(MODE == SWEEP_A ? p.dC : p.dB) + ((size_t)bg * T + t0 + t + e1) * D + 2 * n;
              store_two(dst, (reinterpret_cast<uintptr_t>(dst) & (2 * sizeof(TIn) - 1)) == 0, v_re, v_im, true);
            }
          }
        }
      }
      float v[8];   // [token tile][re, im][token]
#pragma unroll
      for (int tt = 0; tt < 2; ++tt) {
        const float2 r = un2(sre[tt]), i = un2(sim[tt]);
        v[4 * tt] = r.x; v[4 * tt + 1] = r.y; v[4 * tt + 2] = i.x; v[4 * tt + 3] = i.y;
      }
      Scatter<8, 16, 4>::run(v, o.lane);
      red[2 * (((c & 1) * W + o.w) * L + 8 * ((o.lane >> 4) & 1) + 2 * o.q + ((o.lane >> 2) & 1)) + ((o.lane >> 3) & 1)] = v[0];
    }

    // ---- the state behind the chunk --------------------------------------------------------------------------------------
    {
      constexpr int NR = REV ? NY : NI;
      uint32_t op[2][3][4];   // columns of P(L,i) h_i b_i or of conj(a_j) c_j, k = token
#pragma unroll
      for (int tt = 0; tt < 2; ++tt) {
        const int t = 8 * tt + 2 * o.q;
        f2 er, ei;
        if (REV) load_cf2(tab + 2 * t * TABW, 2 * TABW, er, ei);
        else load_cf2(tab + V_KAPPA + 2 * t, 2, er, ei);
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) {
          f2 r, i, xr, xi;
          uint32_t wr[3], wi[3];
          tokens_of(REV ? lay.c : lay.b, grp, tt, r, i);
          if (REV) cmul2_conj_a(er, ei, r, i, xr, xi);
          else cmul2(er, ei, r, i, xr, xi);
          split<3>(xr, wr); split<3>(xi, wi);
#pragma unroll
          for (int k = 0; k < 3; ++k) { op[grp][k][2 * tt] = wr[k]; op[grp][k][2 * tt + 1] = wi[k]; }
        }
      }
      const cf m = load_cf(tab + 2 * nb * TABW);
      const f2 r2 = dup2(m.re), i2 = dup2(REV ? -m.im : m.im), n2 = dup2(REV ? m.im : -m.im);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        uint32_t rows[2][NR][2];   // [pt]
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          uint32_t r[4];
          ldmatrix4<true>(r, (REV ? y_rows(c, k) : u_rows(c, k)) + r_lo + 32 * s);
          rows[0][k][0] = r[0]; rows[0][k][1] = r[1]; rows[1][k][0] = r[2]; rows[1][k][1] = r[3];
        }
        float d[4][4];   // [grp, pt]
        products<4, 3, NR>(d, [&](int t) { return &op[t >> 1][0]; }, [&](int t) { return &rows[t & 1][0]; });
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int grp = t >> 1, k = t & 1;
          const f2 zr = z.re[grp][2 * s + k], zi = z.im[grp][2 * s + k];
          z.re[grp][2 * s + k] = fma2(n2, zi, fma2(r2, zr, mk2(d[t][0], d[t][1])));
          z.im[grp][2 * s + k] = fma2(i2, zr, fma2(r2, zi, mk2(d[t][2], d[t][3])));
        }
      }
    }
    if (c + 1 < nchunks && o.w == 0) products_of(c + 1, next);
    if (MODE != FORWARD && MODE != SWEEP_B) continue;
    __syncthreads();

    // ---- y or dU: the warps' sums, and the chunk's own part S u (S^T dy) ---------------------------------------------------
    {
      using TO = typename std::conditional<MODE == FORWARD, TY, TIn>::type;
      constexpr int NR = MODE == FORWARD ? NI : NY;
      TO* out = reinterpret_cast<TO*>(MODE == FORWARD ? p.Y : p.dU) + ((size_t)bh * T + t0) * P + row0;
      const bool vec = (P & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & (2 * sizeof(TO) - 1)) == 0;
      uint32_t a[3][4];
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        float4 dr = dpart[2 * it * 32 + o.lane], di = dpart[(2 * it + 1) * 32 + o.lane];
#pragma unroll 1
        for (int k = 1; k < W; ++k) {
          const float4 r = dpart[(k * 4 + 2 * it) * 32 + o.lane], i = dpart[(k * 4 + 2 * it + 1) * 32 + o.lane];
          dr.x += r.x; dr.y += r.y; dr.z += r.z; dr.w += r.w;
          di.x += i.x; di.y += i.y; di.z += i.z; di.w += i.w;
        }
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          const int own = 8 * tt + o.g, src = 8 * it + 2 * o.q;   // FORWARD: j = own, i = src; SWEEP_B: i = own, j = src
          const f2 vr = tt ? mk2(dr.z, dr.w) : mk2(dr.x, dr.y), vi = tt ? mk2(di.z, di.w) : mk2(di.x, di.y);
          f2 pr, pi, hr, hi, gr, gi;
          if (MODE == FORWARD) {
            load_cf2(tab + 2 * (own * TABW + src + 1), 2, pr, pi);
            load_cf2(tab + V_H + 2 * src, 2, hr, hi);
          } else {
            load_cf2(tab + 2 * (src * TABW + own + 1), 2 * TABW, pr, pi);
            const cf h1 = load_cf(tab + V_H + 2 * own);
            hr = dup2(h1.re); hi = dup2(h1.im);
          }
          cmul2(pr, pi, hr, hi, gr, gi);
          const cf kc = load_cf(tab + V_KC + 2 * own);
          const float2 s = un2(fma2(neg2(gi), vi, mul2(gr, vr))), v_r = un2(vr), v_i = un2(vi);
          const float g0 = kc.re * v_r.x - kc.im * v_i.x, g1 = kc.re * v_r.y - kc.im * v_i.y;
          const bool m0 = MODE == FORWARD ? src < own : src > own, m1 = MODE == FORWARD ? src + 1 < own : src + 1 > own;
          uint32_t wd[3];
          split<3>(mk2(src == own ? g0 : m0 ? s.x : 0.f, src + 1 == own ? g1 : m1 ? s.y : 0.f), wd);
#pragma unroll
          for (int k = 0; k < 3; ++k) a[k][2 * it + tt] = wd[k];
          if (MODE == SWEEP_B && o.w == 0 && it == tt && o.q == (o.g >> 1)) {
            const cf mn = load_cf(tab + V_MNEXT + 2 * own);
            dd[(c & 1) * L + own] = make_float4(sig[own] * ((o.g & 1) ? v_r.y : v_r.x), -sig[own] * ((o.g & 1) ? v_i.y : v_i.x), mn.re, mn.im);
          }
        }
      }
#pragma unroll 1
      for (int pt = o.w; pt < 8; pt += W) {
        uint32_t rows[NR][2];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          uint32_t r[4];   // (the second pair of tiles is not used)
          ldmatrix4<true>(r, (MODE == FORWARD ? u_rows(c, k) : y_rows(c, k)) + ((o.lane & 15) * PP) + 16 * pt);
          rows[k][0] = r[0]; rows[k][1] = r[1];
        }
        float d[1][4];
        products<1, 3, NR>(d, [&](int) { return &a[0]; }, [&](int) { return &rows[0]; });
        float4 v = part[pt * 32 + o.lane];
#pragma unroll 1
        for (int k = 1; k < W; ++k) {
          const float4 x = part[(k * 8 + pt) * 32 + o.lane];
          v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        if (__any_sync(0xffffffffu, not_finite(d[0][0] + d[0][1]))) {
          d[0][0] = d[0][1] = d[0][2] = d[0][3] = 0.f;
#pragma unroll 1
          for (int i = 0; i < L; ++i) {
            uint32_t one[NR][2];
#pragma unroll
            for (int k = 0; k < NR; ++k)
#pragma unroll
              for (int r = 0; r < 2; ++r) one[k][r] = rows[k][r] & only_token(i, 8 * r + 2 * o.q);
            float e[1][4];
            products<1, 3, NR>(e, [&](int) { return &a[0]; }, [&](int) { return &one[0]; });
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const int own = 8 * (r >> 1) + o.g;
              if (MODE == FORWARD ? i <= own : i >= own) d[0][r] += e[0][r];
            }
          }
        }
        const int pp = 8 * pt + 2 * o.q;
        if (pp < prows) {
          if (o.g < nb) store_two(out + (size_t)o.g * P + pp, vec, v.x + d[0][0], v.y + d[0][1], pp + 1 < prows);
          if (8 + o.g < nb) store_two(out + (size_t)(8 + o.g) * P + pp, vec, v.z + d[0][2], v.w + d[0][3], pp + 1 < prows);
        }
      }
    }
  }

  if (ONLY_STATES) {
    store_tile<true>(z, (REV ? p.gloc : p.zloc) + ((size_t)seg * p.batch * p.heads + bh) * P * D, o, row0, P, N);
    return;
  }
  if (MODE == FORWARD && p.zfinal && seg == p.nseg - 1) store_tile<false>(z, p.zfinal + (size_t)bh * P * D, o, row0, P, N);
  if (!BACK) return;
  __syncthreads();
  finish_scalars(nchunks - 1);
  float* scratch = reinterpret_cast<float*>(smem);   // (the raw rows are done with)
  if (MODE == SWEEP_A && seg == p.nseg - 1) {   // S_T = sum d_final conj(z_final)
    f2 sr = 0ull, si = 0ull;
    if (p.dfinal)
      read_tile<false>(p.dfinal + (size_t)bh * P * D, o, row0, P, N, [&](int r, int i, f2 re, f2 im) {
        sr = fma2(im, z.im[r][i], fma2(re, z.re[r][i], sr));
        si = fma2(neg2(re), z.im[r][i], fma2(im, z.re[r][i], si));
      });
    const float re = warp_sum(hsum(sr)), im = warp_sum(hsum(si));
    if (o.lane == 0) { scratch[2 * o.w] = re; scratch[2 * o.w + 1] = im; }
    __syncthreads();
    if (tid == 0) {
      float a = 0.f, d = 0.f;
      for (int k = 0; k < W; ++k) { a += scratch[2 * k]; d += scratch[2 * k + 1]; }
      put(p.sT + 2 * (size_t)bh, a, p.ptiles > 1); put(p.sT + 2 * (size_t)bh + 1, d, p.ptiles > 1);
    }
  }
  if (MODE == SWEEP_B && seg == 0) {   // z = lambda_0: the start state and the prev-tap of the first token
    if (p.Bprev) {
      const TIn* Bp = reinterpret_cast<const TIn*>(p.Bprev) + (size_t)bg * D;
      const TIn* Up = reinterpret_cast<const TIn*>(p.Uprev) + (size_t)bh * P + row0;
      const cf kp = load_cf(K);
      float* s_du = scratch + 2 * W;   // [W][64]: Re sum conj(kp b_prev) lambda over a warp's columns
      cf dkp = {0.f, 0.f}, x[2];
#pragma unroll
      for (int grp = 0; grp < 2; ++grp) {   // sum over the rows of u_prev lambda, per column
        const int n = 16 * o.w + 8 * grp + o.g;
        f2 sr = 0ull, si = 0ull;
#pragma unroll
        for (int pt = 0; pt < 8; ++pt) {
          const int r = 8 * pt + 2 * o.q;
          const f2 u = mk2(r < prows ? to_f32(Up[r]) : 0.f, r + 1 < prows ? to_f32(Up[r + 1]) : 0.f);
          sr = fma2(u, z.re[grp][pt], sr); si = fma2(u, z.im[grp][pt], si);
        }
        float re = hsum(sr), im = hsum(si);
        re += __shfl_xor_sync(0xffffffffu, re, 1); im += __shfl_xor_sync(0xffffffffu, im, 1);
        re += __shfl_xor_sync(0xffffffffu, re, 2); im += __shfl_xor_sync(0xffffffffu, im, 2);
        const cf bp = n < N ? load_c(Bp, n) : cf{0.f, 0.f};
        x[grp] = cmul(kp, bp);
        if (o.q == 0 && n < N) {
          const cf g = cmul_conj_a(kp, {re, im});
          dkp = cadd(dkp, cmul_conj_a(bp, {re, im}));
          if (p.dBprev) {
            if (p.spread) {
              float* dst = p.dBprev_head + (size_t)bh * D + 2 * n;
              put(dst, g.re, p.ptiles > 1); put(dst + 1, g.im, p.ptiles > 1);
            } else {
              TIn* dst = reinterpret_cast<TIn*>(p.dBprev) + (size_t)bg * D + 2 * n;
              dst[0] = from_f32<TIn>(g.re); dst[1] = from_f32<TIn>(g.im);
            }
          }
        }
      }
      const float re = warp_sum(dkp.re), im = warp_sum(dkp.im);
      if (o.lane == 0) { scratch[2 * o.w] = re; scratch[2 * o.w + 1] = im; }
#pragma unroll
      for (int pt = 0; pt < 8; ++pt) {
        f2 v = 0ull;
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) v = fma2(dup2(x[grp].im), z.im[grp][pt], fma2(dup2(x[grp].re), z.re[grp][pt], v));
        float2 s = un2(v);
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) { s.x += __shfl_xor_sync(0xffffffffu, s.x, m); s.y += __shfl_xor_sync(0xffffffffu, s.y, m); }
        if (o.g == 0) { s_du[o.w * ROWS + 8 * pt + 2 * o.q] = s.x; s_du[o.w * ROWS + 8 * pt + 2 * o.q + 1] = s.y; }
      }
      __syncthreads();
      if (p.dUprev)
        for (int r = tid; r < prows; r += NT) {
          float s = 0.f;
          for (int k = 0; k < W; ++k) s += s_du[k * ROWS + r];
          reinterpret_cast<TIn*>(p.dUprev)[(size_t)bh * P + row0 + r] = from_f32<TIn>(s);
        }
    }
    if (tid == 0) {
      cf dkp = {0.f, 0.f};
      if (p.Bprev)
        for (int k = 0; k < W; ++k) dkp = cadd(dkp, load_cf(scratch + 2 * k));
      put(p.dK + (size_t)bh * T * 4, dkp.re, p.ptiles > 1); put(p.dK + (size_t)bh * T * 4 + 1, dkp.im, p.ptiles > 1);
    }
    if (p.dinit) {
      scale_tile<true>(z, load_cf(M));
      store_tile<false>(z, p.dinit + (size_t)bh * P * D, o, row0, P, N);
    }
  }
}

// grid (heads, batch, ptiles x segments [x the two sweeps])
template <typename TIn, typename TY>
__global__ void __maxnreg__(168) sweep_fwd_kernel(SweepParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  walk<TIn, TY, FORWARD>(p, blockIdx.z % p.ptiles, blockIdx.z / p.ptiles, smem);
}
template <typename TIn, typename TY>
__global__ void __maxnreg__(168) sweep_bwd_kernel(SweepParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int pt = blockIdx.z % p.ptiles, seg = blockIdx.z / p.ptiles;   // the longer sweep first
  if (seg < p.nseg) walk<TIn, TY, SWEEP_B>(p, pt, seg, smem);
  else walk<TIn, TY, SWEEP_A>(p, pt, seg - p.nseg, smem);
}
// where each segment ends from zero: forward segments 0 .. nseg - 2, and for the backward also reverse segments 1 .. nseg - 1
template <typename TIn, typename TY>
__global__ void __maxnreg__(168) segment_kernel(SweepParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int pt = blockIdx.z % p.ptiles, seg = blockIdx.z / p.ptiles;
  if (seg < p.nseg - 1) walk<TIn, TY, STATES>(p, pt, seg, smem);
  else walk<TIn, TY, ADJ_STATES>(p, pt, seg - (p.nseg - 2), smem);
}

// From where the segments end from zero to where they start: the caller's state at that end of the sequence through the
// segments between, in walking order and in place (all in float32).  A thread per (row, column) of the state, 8 segments'
// loads at a time; blockIdx.z 0: the walk forward in time, 1: the adjoint's.  (Folded by every CTA of the sweeps for itself
// this was a chain of up to nseg round trips to L2 in front of each: at (2, 4, 256, N 32) 48 of the forward sweep's 50 us.)
template <typename TIn>
__global__ void __launch_bounds__(256) combine_kernel(SweepParams p) {
  const int e = blockIdx.y * 256 + threadIdx.x, bh = blockIdx.x, N = p.N, D = 2 * N, nseg = p.nseg;
  if (e >= p.P * N) return;
  const bool rev = blockIdx.z != 0;
  const size_t bhs = (size_t)p.batch * p.heads, size = (size_t)p.P * D;
  float* loc = (rev ? p.gloc : p.zloc) + bh * size + 2 * (size_t)e;
  const float* prod = (rev ? p.gprod : p.zprod) + 2 * (size_t)bh;
  const float* init = rev ? p.dfinal : p.z0;
  cf z = {0.f, 0.f};
  if (init) z = {init[bh * size + 2 * (size_t)e], init[bh * size + 2 * (size_t)e + 1]};
  if (!rev) {
    z = cmul(load_cf(p.M + (size_t)bh * p.T * 2), z);
    if (p.Bprev) {   // the prev-tap of the first token
      const int row = e / N, n = e % N, bg = bh / p.heads * p.groups + bh % p.heads / (p.heads / p.groups);
      const cf x = cmul(load_cf(p.K + (size_t)bh * p.T * 4), load_c(reinterpret_cast<const TIn*>(p.Bprev) + (size_t)bg * D, n));
      const float u = to_f32(reinterpret_cast<const TIn*>(p.Uprev)[(size_t)bh * p.P + row]);
      z = {z.re + u * x.re, z.im + u * x.im};
    }
  }
  for (int k0 = 0; k0 < nseg; k0 += 8) {
    cf f[8], m[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      f[k] = m[k] = {0.f, 0.f};
      if (k0 + k < nseg - 1) {   // (nothing starts behind the last segment of the walk)
        const size_t at = (size_t)(rev ? nseg - 1 - (k0 + k) : k0 + k) * bhs;
        f[k] = load_cf(loc + at * size); m[k] = load_cf(prod + 2 * at);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k0 + k >= nseg) break;
      store_cf(loc + (size_t)(rev ? nseg - 1 - (k0 + k) : k0 + k) * bhs * size, z);
      z = cadd(rev ? cmul_conj_a(m[k], z) : cmul(m[k], z), f[k]);
    }
  }
}

// What follows the sweeps, in one launch: dM per (batch, head), and where heads or slices of P were still apart, dB, dC
// and dB_prev from their float32 parts.
constexpr int FINISH = 1024;   // threads
struct FinishParams {
  const float *M, *K, *dK, *sterm, *sT, *dB_head, *dC_head, *dBprev_head;
  float* dM;
  void *dB, *dC, *dBprev;
  int BH, heads, groups, T, N, spread;
};

// One CTA per (batch, head): S_t = S_T + sum_{s >= t} (sterm_s - conj(h_s) dh_s), dM_t = (S_t - conj(kp_t) dkp_t) / conj(m_t).
// 1024 tokens at a time: the turns are serial (256 at a time took 20 us over 4096 tokens).
__device__ void finish_dm(const FinishParams& p) {
  __shared__ double s_wr[FINISH / 32], s_wi[FINISH / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, T = p.T;
  const size_t bh = blockIdx.x;
  const float *st = p.sterm + bh * T * 2, *M = p.M + bh * T * 2, *K = p.K + bh * T * 4, *dK = p.dK + bh * T * 4;
  float* dM = p.dM + bh * T * 2;
  double carry_r = p.sT[bh * 2], carry_i = p.sT[bh * 2 + 1];
  for (int hi = T; hi > 0; hi -= FINISH) {
    const int t = hi - 1 - tid;  // thread 0 owns the latest token of the tile
    double vr = 0.0, vi = 0.0;
    cf m = {0.f, 0.f}, kd = {0.f, 0.f};
    if (t >= 0) {
      cf mn = {1.f, 0.f}, kpn = {0.f, 0.f}, dh;
      m = load_cf(M + 2 * (size_t)t);
      kd = cmul_conj_a(load_cf(K + 4 * (size_t)t), {dK[4 * (size_t)t], dK[4 * (size_t)t + 1]});   // conj(kp) dkp
      const cf kc = load_cf(K + 4 * (size_t)t + 2);
      if (t + 1 < T) {
        mn = load_cf(M + 2 * (size_t)t + 2); kpn = load_cf(K + 4 * (size_t)t + 4);
        dh = {dK[4 * (size_t)t + 4], dK[4 * (size_t)t + 5]};
      } else {
        dh = {dM[2 * (size_t)t], dM[2 * (size_t)t + 1]};   // (left there by the sweep: the last token has no next one)
      }
      const cf r = cmul_conj_a(cadd(cmul(mn, kc), kpn), dh);
      vr = (double)st[2 * t] - r.re; vi = (double)st[2 * t + 1] - r.im;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double ar = __shfl_up_sync(0xffffffffu, vr, o), ai = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) { vr += ar; vi += ai; }
    }
    if (lane == 31) { s_wr[w] = vr; s_wi[w] = vi; }
    __syncthreads();
    vr += carry_r; vi += carry_i;
    for (int k = 0; k < FINISH / 32; ++k) {
      if (k < w) { vr += s_wr[k]; vi += s_wi[k]; }
      carry_r += s_wr[k]; carry_i += s_wi[k];
    }
    if (t >= 0) {
      const float den = m.re * m.re + m.im * m.im;
      // S / conj(m) = S * m / |m|^2
      float outr = 0.f, outi = 0.f;
      if (den > 0.f) {
        const double sr = vr - kd.re, si = vi - kd.im, inv = 1.0 / (double)den;
        outr = (float)((sr * m.re - si * m.im) * inv);
        outi = (float)((sr * m.im + si * m.re) * inv);
      }
      dM[2 * t] = outr; dM[2 * t + 1] = outi;
    }
    __syncthreads();
  }
}
// a thread per complex column of a row of dB / dC
template <typename TIn>
__device__ __forceinline__ void finish_columns(const FinishParams& p, unsigned block) {
  const int hpg = p.heads / p.groups, N = p.N, D = 2 * N;
  const size_t i = (size_t)block * FINISH + threadIdx.x, rows = (size_t)(p.BH / p.heads) * p.groups * p.T;
  if (i >= rows * N) return;
  const size_t row = i / N, n = i % N, bg = row / p.T, t = row % p.T;
  const size_t bh0 = bg / p.groups * p.heads + bg % p.groups * hpg;
  auto sum_heads = [&](const float* src, size_t stride, void* out, size_t at) {
    cf v = {0.f, 0.f};
    for (int h = 0; h < hpg; ++h) v = cadd(v, {src[h * stride], src[h * stride + 1]});
    TIn* dst = reinterpret_cast<TIn*>(out) + at;
    dst[0] = from_f32<TIn>(v.re); dst[1] = from_f32<TIn>(v.im);
  };
  sum_heads(p.dB_head + (bh0 * p.T + t) * D + 2 * n, (size_t)p.T * D, p.dB, row * D + 2 * n);
  sum_heads(p.dC_head + (bh0 * p.T + t) * D + 2 * n, (size_t)p.T * D, p.dC, row * D + 2 * n);
  if (t == 0 && p.dBprev) sum_heads(p.dBprev_head + bh0 * D + 2 * n, D, p.dBprev, bg * D + 2 * n);
}
template <typename TIn>
__global__ void __launch_bounds__(FINISH) bwd_finish_kernel(FinishParams p) {
  if (blockIdx.x < (unsigned)p.BH) finish_dm(p);
  else finish_columns<TIn>(p, blockIdx.x - p.BH);
}

struct SimtConfig {
  int W, ptiles, nseg, seg_len;
};

template <typename TIn, typename TY>
size_t smem_of(int W, Mode mode) { return (size_t)Layout(W, sizeof(TIn), sizeof(TY), Parts<TIn>::N, Parts<TY>::N, mode).bytes; }

// Segments of T.  The model counts the time of the most loaded SM in chunks of a full one: it holds ``fit`` CTAs at a time
// (168 registers a thread and shared memory) and is slowed by latency when it holds fewer; measured per chunk of the forward
// sweep with N = 48: 4.6, 5.9, 7.3 and 8.2 us for 1 to 4 CTAs.  A split adds a pre-pass (0.37 of a chunk per chunk), two launches
// (1 chunk) and the combination's traffic.  Sequences up to 64 tokens stay whole.  Forward + backward by segments, us:
// (16, 4, 2048, N 48 fp16) 1: 1650, 4: 831, 9: 647, 16: 669, 32: 698; (16, 32, 1024, N 32 bf16) 1: 1301, 4: 1359, 16: 1509;
// (2, 4, 256, N 32 fp32) 1: 242, 4: 98, 16: 48.
void plan_segments(const ScanDims& d, SimtConfig& c) {
  c.nseg = 1; c.seg_len = d.T;
  if (d.T <= 64) return;
  const int fit = c.W == 1 ? 5 : c.W <= 3 ? 4 : c.W == 4 ? 2 : 1;
  const long long ctas = (long long)d.batch * d.heads * c.ptiles;
  auto load = [&](long long n) {
    const long long q = (n + 147) / 148;
    return (double)(q / fit) + (q % fit ? 0.42 + 0.58 * (double)(q % fit) / fit : 0.0);
  };
  double best = (d.T + L - 1) / L * load(ctas);
  for (int n = 2, last = 0; n <= 64 && last != 1; ++n) {
    const int chunks = ((d.T + n - 1) / n + L - 1) / L, len = chunks * L, segs = (d.T + len - 1) / len;
    if (segs < 2) break;
    if (chunks == last) continue;
    last = chunks;
    const double cost = chunks * (load(ctas * segs) + 0.37 * load(ctas * (segs - 1))) + 1.0 + 3e-4 * (double)(ctas * segs * c.W);
    if (cost < 0.97 * best) { best = cost; c.nseg = segs; c.seg_len = len; }
  }
}

bool make_config(const ScanDims& d, SimtConfig& c) {
  if (d.N < 1 || d.N > 128 || d.P < 1) return false;
  c.W = (d.N + 15) / 16;
  c.ptiles = (d.P + ROWS - 1) / ROWS;
  plan_segments(d, c);
  return true;
}

SweepParams base_params(const void* U, const float* M, const float* K, const void* B,
                        const void* C, const float* z0, const void* Bprev, const void* Uprev,
                        const ScanDims& d, const SimtConfig& c) {
  SweepParams p{};
  p.U = U; p.B = B; p.C = C; p.Bprev = Bprev; p.Uprev = Uprev; p.M = M; p.K = K; p.z0 = z0;
  p.batch = d.batch; p.heads = d.heads; p.groups = d.groups; p.T = d.T; p.P = d.P; p.N = d.N;
  p.W = c.W; p.ptiles = c.ptiles; p.nseg = c.nseg; p.seg_len = c.seg_len;
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

constexpr size_t SIMT_SMEM_MAX = 200 * 1024;
static_assert(Layout(8, 4, 4, 3, 3, SWEEP_B).bytes <= (int)SIMT_SMEM_MAX, "the widest state fits");

template <typename TIn, typename TY>
int launch_sweeps(const SweepParams& p, const SimtConfig& c, bool bwd, cudaStream_t st) {
  auto pre = segment_kernel<TIn, TY>;
  auto k = bwd ? sweep_bwd_kernel<TIn, TY> : sweep_fwd_kernel<TIn, TY>;
  static std::atomic<unsigned long long> done[3];
  if (int e = ensure_smem(k, SIMT_SMEM_MAX, done[bwd])) return e;
  if (int e = c.nseg > 1 ? ensure_smem(pre, SIMT_SMEM_MAX, done[2]) : SL_OK) return e;
  const unsigned dirs = bwd ? 2 : 1;
  if (c.nseg > 1) {
    pre<<<dim3(p.heads, p.batch, dirs * (c.nseg - 1) * c.ptiles), 32 * c.W, std::max(smem_of<TIn, TY>(c.W, STATES), smem_of<TIn, TY>(c.W, ADJ_STATES)), st>>>(p);
    combine_kernel<TIn><<<dim3((unsigned)p.batch * p.heads, (unsigned)(p.P * p.N + 255) / 256, dirs), 256, 0, st>>>(p);
    note_launches(2);
  }
  k<<<dim3(p.heads, p.batch, dirs * c.nseg * c.ptiles), 32 * c.W, bwd ? smem_of<TIn, TY>(c.W, SWEEP_B) : smem_of<TIn, TY>(c.W, FORWARD), st>>>(p);
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
  SL_DISPATCH_DTYPE(io_dtype, TIn, SL_DISPATCH_DTYPE(y_dtype, TY, { rc = launch_sweeps<TIn, TY>(p, c, false, st); }));
  return rc;
}

// heads or slices of P are summed by the last launch
bool spread_of(const ScanDims& d) { return d.groups != d.heads || d.P > ROWS; }

// workspace layout: sterm (batch*heads*T*2) | sT (batch*heads*2) | where spread: dB | dC (each batch*heads*T*2N floats) |
//                   dB_prev (batch*heads*2N) | the segments of the two sweeps
size_t scan_simt_bwd_workspace(const ScanDims& d) {
  const size_t bh = (size_t)d.batch * d.heads, bht = bh * d.T, D = 2 * (size_t)d.N;
  return round_up(4 * (bht * 2 + bh * 2 + (spread_of(d) ? 2 * bht * D + bh * D : 0)), 256);
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
  const size_t bh = (size_t)d.batch * d.heads, bht = bh * d.T, D = 2 * (size_t)d.N;
  SweepParams p = base_params(U, M, K, B, C, z0, Bprev, Uprev, d, c);
  p.dY = dY; p.dfinal = dfinal;
  p.sterm = reinterpret_cast<float*>(ws);
  p.sT = p.sterm + bht * 2;
  p.dB_head = p.sT + bh * 2; p.dC_head = p.dB_head + bht * D; p.dBprev_head = p.dC_head + bht * D;
  p.spread = spread_of(d);
  p.dU = dU; p.dB = dB; p.dC = dC; p.dK = dK; p.dM = dM; p.dUprev = dUprev; p.dBprev = dBprev; p.dinit = dinit;
  if (c.ptiles > 1) {  // partial sums of the P tiles are accumulated atomically
    if (cudaMemsetAsync(ws, 0, need, st) != cudaSuccess || cudaMemsetAsync(dK, 0, bht * 16, st) != cudaSuccess ||
        cudaMemsetAsync(dM, 0, bht * 8, st) != cudaSuccess)
      return SL_ERR_LAUNCH_FAILED;
  }
  float* segments = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + need);
  segment_scratch(d, c, segments, &p.zloc, &p.zprod);
  segment_scratch(d, c, segments + segment_floats(d, c), &p.gloc, &p.gprod);
  int rc = SL_ERR_UNSUPPORTED;
  SL_DISPATCH_DTYPE(io_dtype, TIn, SL_DISPATCH_DTYPE(dy_dtype, TY, { rc = launch_sweeps<TIn, TY>(p, c, true, st); }));
  if (rc != SL_OK) return rc;
  FinishParams f{};
  f.M = M; f.K = K; f.dK = dK; f.sterm = p.sterm; f.sT = p.sT; f.dB_head = p.dB_head; f.dC_head = p.dC_head;
  f.dBprev_head = p.dBprev_head; f.dM = dM; f.dB = dB; f.dC = dC; f.dBprev = Bprev ? dBprev : nullptr;
  f.BH = (int)bh; f.heads = d.heads; f.groups = d.groups; f.T = d.T; f.N = d.N;
  const size_t columns = p.spread ? (size_t)d.batch * d.groups * d.T * d.N : 0;
  const unsigned blocks = (unsigned)(bh + (columns + FINISH - 1) / FINISH);
  SL_DISPATCH_DTYPE(io_dtype, TIn, { bwd_finish_kernel<TIn><<<blocks, FINISH, 0, st>>>(f); });
  note_launches(1);
  return launch_status();
}

}  // namespace sl
