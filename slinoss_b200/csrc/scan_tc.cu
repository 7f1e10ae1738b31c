// Chunked v2x2ssd scan on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// Supported: P = 64, N = 64 or 128 (blocks of 64 oscillators, 128 real columns), bf16 or fp16 operands, float32 state.
// Everything else takes the float32 path.  (Narrower N would fit with zero columns and run 4 times faster than
// there, fp16 forward + backward of 64 streams x 2048 tokens x N = 48: 174 against 663 us; but the products round
// their operands to 16 bits and need every |m| > 0, which the float32 sweeps do not.)
//
// Formulation (per (batch, head); chunk of L = 64 tokens, local index t, s).  The two
// taps are merged into one source coefficient with a one-token look-ahead,
//     g_s = kc_s + kp_{s+1} / m_{s+1},
// and the carried state is W = z + u (x) (kp_next / m_next) b, which obeys the
// single-tap recurrence  W_s = m_s W_{s-1} + u_s (x) (g_s b_s)  with
//     y_t = Re<c_t, W_t> - u_t Re(conj(c_t) (g_t - kc_t) b_t).
// With the in-chunk prefix  Pi_t = prod_{s<=t} m_s = exp(l_t) phi_t  (l = cumulative
// log|m|, |phi| = 1) the chunk is four real GEMMs over the interleaved (re, im) lanes:
//     Q_t   = conj(c_t) phi_t                       (unit rotation of C, in place)
//     K'_s  = conj(phi_s) g_s b_s                   (in place over B, stored conjugated)
//     S     = mask_{s<t}( (Q K'^T) * exp(l_t - l_s) ),  S_tt = Re(conj(c_t) kc_t b_t)
//     Y     = S U + exp(l_t) * (Q Zv^T)             (Zv = conj of the chunk-start state)
//     Zv'   = conj(phi_end) (exp(l_end) Zv + (exp(l_end - l_s) U)^T K')
// Magnitudes only ever enter as exp(non-positive), exactly like the reference's
// chunk_scan policy (slinoss/ops/v2x2ssd/reference.py:498-523, 1224-1261); phases are
// applied to the 16-bit operands, decays to float32 accumulators.
//
// A stream is walked chunk by chunk by one CTA; streams that do not fill the chip are split into segments of
// chunks: a cheap pre-pass over the segments (states only) and a fold (in the sweeps, or a combine kernel for many
// segments) give every segment its start state, and the segments then run side by side.  scan_tc_fwd.cuh and scan_tc_bwd.cuh describe the kernels and
// the thread-to-data mappings; plan_segments() below holds the rule for the split.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "common.cuh"
#include "host_abi.h"
#include "tc_common.cuh"

namespace sl {
namespace {

using namespace tc;

constexpr int L = 64;
constexpr uint32_t TILE = 8192;           // one [64][128 B] tile

__device__ int g_tc_status = 0;

template <typename T> struct Pack2;
template <> struct Pack2<__nv_bfloat16> {
  static __device__ __forceinline__ float2 unpack(uint32_t v) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v));
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  // two words (re, im), (re, im) -> the pair of real parts and the pair of imaginary parts, and back
  static __device__ __forceinline__ void split(uint32_t w0, uint32_t w1, f2& re, f2& im) {
    re = mk2(__uint_as_float(w0 << 16), __uint_as_float(w1 << 16));
    im = mk2(__uint_as_float(w0 & 0xffff0000u), __uint_as_float(w1 & 0xffff0000u));
  }
  static __device__ __forceinline__ void join(f2 re, f2 im, uint32_t& w0, uint32_t& w1) {
    const float2 a = un2(re), b = un2(im);
    w0 = pack(a.x, b.x); w1 = pack(a.y, b.y);
  }
  static __device__ __forceinline__ f2 natural(uint32_t w) {
    return mk2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  static __device__ __forceinline__ uint32_t pack2(f2 v) { const float2 a = un2(v); return pack(a.x, a.y); }
  static constexpr int fmt = 1;
};
template <> struct Pack2<__half> {
  static __device__ __forceinline__ float2 unpack(uint32_t v) {
    return __half22float2(*reinterpret_cast<__half2*>(&v));
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ void split(uint32_t w0, uint32_t w1, f2& re, f2& im) {
    const float2 a = unpack(w0), b = unpack(w1);
    re = mk2(a.x, b.x); im = mk2(a.y, b.y);
  }
  static __device__ __forceinline__ void join(f2 re, f2 im, uint32_t& w0, uint32_t& w1) {
    const float2 a = un2(re), b = un2(im);
    w0 = pack(a.x, b.x); w1 = pack(a.y, b.y);
  }
  static __device__ __forceinline__ f2 natural(uint32_t w) { const float2 a = unpack(w); return mk2(a.x, a.y); }
  static __device__ __forceinline__ uint32_t pack2(f2 v) { const float2 a = un2(v); return pack(a.x, a.y); }
  static constexpr int fmt = 0;
};

__device__ __forceinline__ void report_timeout(int code) { atomicCAS(&g_tc_status, 0, code); }

// Limit of the kernels' bounded waits in SM clocks: about a second by default; the environment
// variable SLINOSS_B200_WAIT_CLOCKS (read at every launch) overrides it, which is how the test of
// the unwind path makes a wait expire without anything being wrong.
static long long wait_limit_clocks() {
  if (const char* e = getenv("SLINOSS_B200_WAIT_CLOCKS")) {
    const long long v = atoll(e);
    if (v > 0) return v;
  }
  return tc::WAIT_CLOCKS_DEFAULT;
}

// A wait that did not succeed at once: true when the barrier flips within ``limit`` SM clocks, false as soon as
// another wait of the CTA has expired (``abort_flag``) or when this one does (recorded).
__device__ __noinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, long long limit, int* abort_flag, int code) {
  const long long t_begin = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*reinterpret_cast<volatile int*>(abort_flag)) return false;
    if (clock64() - t_begin > limit) {
      report_timeout(code);
      *reinterpret_cast<volatile int*>(abort_flag) = 1;
      return false;
    }
  }
  return true;
}

// coefficient of the pending prev-tap of the token before the sequence: kp_0 / m_0
__device__ __forceinline__ void pending_tap(const float* Mb, const float* Kb, float& xr, float& xi) {
  const float mr = Mb[0], mi = Mb[1], kr = Kb[0], ki = Kb[1];
  const float den = mr * mr + mi * mi;
  xr = (kr * mr + ki * mi) / den;
  xi = (ki * mr - kr * mi) / den;
}

// Per-chunk scalars, computed by one warp (two tokens per lane) with shuffle scans.  Layout of a table (floats):
//  [0, 256)    per token: phi_t (re, im), w_t = conj(phi_t) g_t (re, im)
//  [256, 512)  per token: kc_t (re, im), exp(l_t), exp(l_end - l_t)
//  [512, 576)  per token: l_t in units of log 2
//  [576, 579)  exp(l_end), unit phase of Pi_end (re, im)
//  forward only:
//  [592, 848)  per block q of 16 tokens and token s < 16 q: exp(l_{16 q} - l_s)
//  [848, 912)  per token: exp(l_t - l_{16 (t / 16)})
// A decay factor exp(l_t - l_s), s < t, is a product of the last two outside the 16 x 16 blocks on the diagonal
// (both factors are <= 1, so nothing can overflow): the masking epilogue needs one multiplication per cell there
// instead of an exponential.  (The backward's masking epilogue runs in the shadow of its MMAs: there the plain
// exponentials measured 4 % faster than the branch on the block's place.)
constexpr int SC_KCL = 256, SC_L2 = 512, SC_TAIL = 576, SC_COL = 592, SC_ROW = 848, SCW = 912, SCW_B = 592;
struct ScalarRaw { float2 m[3]; float4 k[3]; };   // a lane's two tokens and the one after them
__device__ __forceinline__ ScalarRaw load_scalars(const float* __restrict__ Mb, const float* __restrict__ Kb, int t0,
                                                  int T, int lane) {
  ScalarRaw r;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int t = t0 + 2 * lane + q;
    r.m[q] = make_float2(1.f, 0.f);
    r.k[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < T) {
      r.m[q] = *reinterpret_cast<const float2*>(Mb + 2 * (size_t)t);
      r.k[q] = *reinterpret_cast<const float4*>(Kb + 4 * (size_t)t);
    }
  }
  return r;
}
template <bool FACTORS>
__device__ __forceinline__ void chunk_scalars(float* sc, const ScalarRaw& raw, int lane) {
  const float mr[3] = {raw.m[0].x, raw.m[1].x, raw.m[2].x}, mi[3] = {raw.m[0].y, raw.m[1].y, raw.m[2].y};
  const float kpr[3] = {raw.k[0].x, raw.k[1].x, raw.k[2].x}, kpi[3] = {raw.k[0].y, raw.k[1].y, raw.k[2].y};
  const float kcr[2] = {raw.k[0].z, raw.k[1].z}, kci[2] = {raw.k[0].w, raw.k[1].w};
  // local prefixes over the lane's two tokens
  const float q0 = mr[0] * mr[0] + mi[0] * mi[0], q1 = mr[1] * mr[1] + mi[1] * mi[1];
  const float i0 = rsqrtf(q0), i1 = rsqrtf(q1);
  const float a0 = 0.5f * lg2f(q0), a1 = 0.5f * lg2f(q1);
  const float u0r = mr[0] * i0, u0i = mi[0] * i0, u1r = mr[1] * i1, u1i = mi[1] * i1;
  float lsum = a0 + a1;                       // inclusive scan of log-magnitudes
  float pr = u0r * u1r - u0i * u1i, pi = u0r * u1i + u0i * u1r;  // and of unit phases
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float ol = __shfl_up_sync(0xffffffffu, lsum, o);
    const float opr = __shfl_up_sync(0xffffffffu, pr, o), opi = __shfl_up_sync(0xffffffffu, pi, o);
    if (lane >= o) {
      lsum += ol;
      const float nr = pr * opr - pi * opi, ni = pr * opi + pi * opr;
      pr = nr; pi = ni;
    }
  }
  float el = __shfl_up_sync(0xffffffffu, lsum, 1);
  float epr = __shfl_up_sync(0xffffffffu, pr, 1), epi = __shfl_up_sync(0xffffffffu, pi, 1);
  if (lane == 0) { el = 0.f; epr = 1.f; epi = 0.f; }
  const float l_end = __shfl_sync(0xffffffffu, lsum, 31);
  float lt[2], phr[2], phi[2];
  lt[0] = el + a0; lt[1] = el + a0 + a1;
  phr[0] = epr * u0r - epi * u0i; phi[0] = epr * u0i + epi * u0r;
  phr[1] = phr[0] * u1r - phi[0] * u1i; phi[1] = phr[0] * u1i + phi[0] * u1r;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float n = rsqrtf(phr[q] * phr[q] + phi[q] * phi[q]);
    phr[q] *= n; phi[q] *= n;
    // g = kc + kp_next / m_next
    const float den = mr[q + 1] * mr[q + 1] + mi[q + 1] * mi[q + 1];
    const float gr = kcr[q] + (kpr[q + 1] * mr[q + 1] + kpi[q + 1] * mi[q + 1]) / den;
    const float gi = kci[q] + (kpi[q + 1] * mr[q + 1] - kpr[q + 1] * mi[q + 1]) / den;
    const int i = 2 * lane + q;
    reinterpret_cast<float4*>(sc)[i] =
        make_float4(phr[q], phi[q], phr[q] * gr + phi[q] * gi, phr[q] * gi - phi[q] * gr);   // phi, conj(phi) g
    reinterpret_cast<float4*>(sc + SC_KCL)[i] = make_float4(kcr[q], kci[q], ex2f(lt[q]), ex2f(l_end - lt[q]));
    sc[SC_L2 + i] = lt[q];
  }
  if constexpr (FACTORS) {
    float lref[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      lref[q] = __shfl_sync(0xffffffffu, lt[0], 8 * q);
      *reinterpret_cast<float2*>(sc + SC_COL + 64 * q + 2 * lane) =
          make_float2(ex2f(fminf(lref[q] - lt[0], 0.f)), ex2f(fminf(lref[q] - lt[1], 0.f)));
    }
    const float lr = lane < 8 ? lref[0] : lane < 16 ? lref[1] : lane < 24 ? lref[2] : lref[3];
    *reinterpret_cast<float2*>(sc + SC_ROW + 2 * lane) = make_float2(ex2f(fminf(lt[0] - lr, 0.f)), ex2f(fminf(lt[1] - lr, 0.f)));
  }
  if (lane == 31) {
    sc[SC_TAIL] = ex2f(l_end);
    sc[SC_TAIL + 1] = phr[1]; sc[SC_TAIL + 2] = phi[1];
  }
}

// Loads and table in one out-of-line call (the backward: its code is long enough for the instruction cache to matter).
__device__ __noinline__ void chunk_scalars_at(float* sc, const float* __restrict__ Mb, const float* __restrict__ Kb,
                                              int t0, int T, int lane) {
  chunk_scalars<false>(sc, load_scalars(Mb, Kb, t0, T, lane), lane);
}

#include "scan_tc_fwd.cuh"
#include "scan_tc_bwd.cuh"

}  // namespace

bool scan_tc_supported(const ScanDims& d, int io_dtype) {
  return d.P == 64 && (d.N == 64 || d.N == 128) && (io_dtype == SL_BF16 || io_dtype == SL_F16) && d.T >= 1 &&
         tc::encode_tiled_fn() != nullptr;
}

namespace {

inline int blocks_of(const ScanDims& d) { return d.N / 64; }
inline int chunks_of(const ScanDims& d) { return (d.T + L - 1) / L; }

// Encoding a tensor map is a driver call and needs a current context, which a thread that has only been told its
// device (an autograd worker, say) may not have yet: the runtime makes one current on the first cudaSetDevice.
void ensure_context() {
  static thread_local int ready = -1;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev != ready && cudaSetDevice(dev) == cudaSuccess) ready = dev;
}

// Splitting in time.  ``streams`` CTAs of ``nchunks`` serial chunks each leave most of the chip idle when there
// are few of them.  With S segments the main kernel runs S * streams CTAs of ceil(nchunks / S) chunks, at the
// price of the pre-pass over the segments (``pre`` of a main chunk per chunk) and of two more launches
// (``fixed`` chunk times).  The model below counts the chunk times of the most loaded SM: an SM with one
// resident CTA takes 1 per chunk, one with two takes ``pair`` (2 when only one fits).
constexpr int FOLD_SEGS = 8;
struct SegPlan { int nseg, cps, tail, whole; };   // tail, whole: see bwd_plan
struct SegCost { double pair, pre, fixed; };
constexpr int SMS = 148;
inline double load_time(long long ctas, double chunks, double pair) {
  const long long per_sm = (ctas + SMS - 1) / SMS;
  return chunks * ((per_sm / 2) * pair + (per_sm & 1));
}
inline SegPlan plan_segments(long long streams, int nchunks, const SegCost& c, double* cost = nullptr) {
  SegPlan best{1, nchunks, 0, 0};
  double t_best = load_time(streams, nchunks, c.pair);
  for (int s = 2; s <= nchunks && s * streams <= 4 * SMS; ++s) {
    const int cps = (nchunks + s - 1) / s, ns = (nchunks + cps - 1) / cps;
    if (ns != s) continue;
    const double t = load_time(streams * s, cps, c.pair) + c.pre * load_time(streams * (s - 1), cps, c.pair) + c.fixed;
    if (t < 0.97 * t_best) { t_best = t; best = {s, cps, 0, 0}; }
  }
  if (cost) *cost = t_best;
  return best;
}
inline SegPlan fwd_plan(const ScanDims& d) {
  return plan_segments((long long)d.batch * d.heads, chunks_of(d),
                       blocks_of(d) == 1 ? SegCost{1.6, 0.5, 4.5} : SegCost{2.0, 0.4, 3.0});
}
// The reverse sweep holds one CTA per SM, so its last round of CTAs leaves SMs idle (20 of 148 with 128 streams, 40 in the
// second round of 256).  There the streams of that round give their last ``tail`` chunks to the idle SMs: these CTAs come
// last in the grid and need nothing of the others, while the rest of a stream waits for the pre-pass over its tail only.
// An idle SM takes ``fill`` tails one after the other, each with 0.7 of a chunk to start up, beside the nC - tail chunks of the
// rest.  The pre-pass takes 0.25 of a chunk per chunk and 1.0 for its launch.  Sweep and pre-pass, us, whole against so split:
// 128 streams x 64 chunks 297 / 280 (tail 7; 8: 297, 4: 291), 256 x 32 301 / 285 (7), 100 x 64 291 (in two equal segments) / 256
// (16), 64 x 64 of two column blocks 297 / 285 (7).
inline SegPlan bwd_plan(const ScanDims& d) {
  const int nb = blocks_of(d), nC = chunks_of(d);
  const long long streams = (long long)d.batch * d.heads, ctas = streams * nb;
  double best;
  const SegPlan plan = plan_segments(ctas, nC, SegCost{2.0, 0.25, 2.0}, &best);
  const int rounds = (int)(ctas / SMS), over = (int)(ctas % SMS);
  if (!over) return plan;
  const int fill = (over + SMS - over - 1) / (SMS - over), tail = (int)((nC - 0.7 * fill) / (fill + 1));
  if (tail < 1 || rounds * (double)nC + (nC - tail) + 0.25 * tail + 1.3 >= 0.98 * best) return plan;
  return {2, nC - tail, tail, (int)((long long)rounds * SMS / nb)};
}
struct SegLayout { size_t seg, pi, total; };
inline SegLayout seg_layout(const ScanDims& d, int nseg) {
  const size_t BH = (size_t)d.batch * d.heads;
  SegLayout o{};
  if (nseg == 1) return o;
  o.pi = round_up(BH * nseg * 64 * 128 * blocks_of(d) * 4, 256);
  o.total = o.pi + round_up(BH * nseg * 8, 256);
  return o;
}

template <typename TIn, typename TY, int MODE, int NB, int NWQ>
int launch_fwd_variant(const TcFwdParams& p, dim3 grid, cudaStream_t st) {
  // Behind a pre-pass (launched behind all that came before, so the operands are there) or its combination: start up while it
  // runs; the state of the segment is waited for where it is read.  A prompt of 16383 tokens x 16 heads 109.6 -> 107.8 us, of
  // 1021 through a mixer 121.3 -> 118.1; the reverse sweep, whose CTAs do not fit beside a pre-pass, gained nothing.
  auto k = scan_tc_fwd_kernel<TIn, TY, MODE, NB, NWQ>;
  constexpr size_t bytes = FwdSmem<NB, MODE == 0, NWQ>::BYTES;
  static std::atomic<unsigned long long> done{0};
  if (int e = ensure_smem(k, bytes, done)) return e;
  if (launch_chained(k, grid, 128 * NWQ + 64, bytes, st, p.from_seg != 0, p) != SL_OK) return SL_ERR_LAUNCH_FAILED;
  note_launches(1);
  return launch_status();
}
// NB = 1: 16 worker warps shorten the chain of a chunk when no SM gets two CTAs, 8 let two CTAs share an SM
template <typename TIn, typename TY, int MODE>
int launch_fwd_kernel(const TcFwdParams& p, dim3 grid, int nb, cudaStream_t st) {
  if (nb == 2) return launch_fwd_variant<TIn, TY, MODE, 2, 4>(p, grid, st);
  if ((long long)grid.x * grid.y <= SMS) return launch_fwd_variant<TIn, TY, MODE, 1, 4>(p, grid, st);
  return launch_fwd_variant<TIn, TY, MODE, 1, 2>(p, grid, st);
}

// pre-pass over the segments: MODE 1 forward in time over (U, B), MODE 2 backwards over (dY, C)
template <typename TIn, int MODE>
int launch_prepass(TcFwdParams p, int BH, int nb, cudaStream_t st) {
  p.to_seg = 1; p.from_seg = 0;
  p.states16 = nullptr; p.zfinal = nullptr; p.z0 = nullptr; p.Bprev = nullptr; p.Uprev = nullptr;
  p.seg0 = MODE == 2 ? 1 : 0;   // the segment that ends the walk contributes to no other
  const dim3 grid((unsigned)BH, (unsigned)(p.nseg - 1));
  return launch_fwd_kernel<TIn, float, MODE>(p, grid, nb, st);
}

// Forward (Y given) or chunk-start / final states only (Y null).
template <typename TIn>
int run_fwd(TcFwdParams& p, const ScanDims& d, int y_dtype, cudaStream_t st) {
  const int BH = d.batch * d.heads, nb = blocks_of(d);
  if (p.nseg > 1) {
    if (int e = launch_prepass<TIn, 1>(p, BH, nb, st)) return e;
    p.from_seg = p.nseg > FOLD_SEGS ? 1 : 2;
  }
  if (p.from_seg == 1) {
    if (launch_chained(scan_tc_combine_kernel<TIn, false>, dim3((unsigned)BH, 16u * nb), 256, 0, st, true, p.seg, (const float2*)p.seg_pi,
                       p.z0, reinterpret_cast<const TIn*>(p.Bprev), reinterpret_cast<const TIn*>(p.Uprev), p.M, p.K, d.heads, d.groups,
                       d.T, d.N, p.nseg) != SL_OK)
      return SL_ERR_LAUNCH_FAILED;
    note_launches(1);
  }
  const dim3 grid((unsigned)BH, (unsigned)p.nseg);
  if (!p.Y)
    return launch_fwd_kernel<TIn, float, 1>(p, grid, nb, st);
  int rc = SL_ERR_UNSUPPORTED;
  SL_DISPATCH_DTYPE(y_dtype, TY, { rc = launch_fwd_kernel<TIn, TY, 0>(p, grid, nb, st); });
  return rc;
}

int scan_tc_fwd_impl(const void* U, const float* M, const float* K, const void* B, const void* C, const float* z0,
                     const void* Bprev, const void* Uprev, void* Y, float* zfinal, void* states16,
                     const ScanDims& d, const SegPlan& plan, uint8_t* seg_ws, int io_dtype, int y_dtype,
                     cudaStream_t st, const ScanLast* last = nullptr) {
  TcFwdParams p{};
  ensure_context();
  const bool bf = io_dtype == SL_BF16;
  const uint64_t BH = (uint64_t)d.batch * d.heads, BG = (uint64_t)d.batch * d.groups, W = 2 * (uint64_t)d.N;
  if (!tc::make_tmap_3d(&p.tmU, U, 64, d.T, BH, 64, bf) || !tc::make_tmap_3d(&p.tmB, B, W, d.T, BG, 64, bf) ||
      (C && !tc::make_tmap_3d(&p.tmC, C, W, d.T, BG, 64, bf)))
    return SL_ERR_LAUNCH_FAILED;
  p.M = M; p.K = K; p.z0 = z0; p.Bprev = Bprev; p.Uprev = Uprev; p.Y = Y; p.zfinal = zfinal;
  p.states16 = states16;
  if (last) { p.state_last = last->state; p.B_last = last->B; p.U_last = last->U; p.U = U; p.B = B; }
  p.heads = d.heads; p.groups = d.groups; p.T = d.T; p.nchunks = chunks_of(d);
  p.nseg = plan.nseg; p.cps = plan.cps;
  if (plan.nseg > 1) {
    const SegLayout lay = seg_layout(d, plan.nseg);
    p.seg = reinterpret_cast<float*>(seg_ws + lay.seg);
    p.seg_pi = reinterpret_cast<float2*>(seg_ws + lay.pi);
  }
  p.wait_limit = wait_limit_clocks();
  if (Y && y_dtype != SL_F32 && !tc::make_tmap_3d(&p.tmY, Y, 64, d.T, BH, 64, y_dtype == SL_BF16))
    return SL_ERR_LAUNCH_FAILED;
  if (states16 && !tc::make_tmap_3d(&p.tmS, states16, 128, (uint64_t)p.nchunks * 64, BH * blocks_of(d), 64, bf))
    return SL_ERR_LAUNCH_FAILED;
  return bf ? run_fwd<__nv_bfloat16>(p, d, y_dtype, st) : run_fwd<__half>(p, d, y_dtype, st);
}

// backward workspace (the carried-tap regions are always reserved: the workspace query does not know whether the
// call will carry B_prev / U_prev)
struct TcBwdLayout {
  size_t states, zfinal, dg, sterm, dkcd, anchor, dbh, dch, dstart, dgb, du2, segs, total;
};
TcBwdLayout tc_bwd_layout(const ScanDims& d) {
  const size_t BH = (size_t)d.batch * d.heads, nC = chunks_of(d), NB = blocks_of(d), W = 2 * (size_t)d.N;
  TcBwdLayout o{};
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t r = off; off += round_up(bytes, 256); return r; };
  o.states = take(BH * nC * 64 * 128 * NB * 2);
  o.zfinal = take(BH * 64 * W * 4);
  o.dg = take(NB * BH * d.T * 8);
  o.sterm = take(NB * BH * d.T * 8);
  o.dkcd = take(NB * BH * d.T * 8);
  o.anchor = take(NB * BH * nC * 8);
  if (d.groups != d.heads) {   // per-head dB / dC (16-bit) before the reduction over the heads of a group
    o.dbh = take(BH * d.T * W * 2);
    o.dch = take(BH * d.T * W * 2);
  }
  o.dstart = take(BH * 64 * W * 4);   // adjoint of the start state when the caller wants no d_initial
  o.dgb = take(BH * 8);               // gradient of the pending tap's coefficient
  if (NB == 2) o.du2 = take(BH * d.T * 64 * 2);   // dU of the second column block
  o.segs = take(std::max(seg_layout(d, fwd_plan(d).nseg).total, seg_layout(d, bwd_plan(d).nseg).total));
  o.total = off;
  return o;
}

}  // namespace

size_t scan_tc_fwd_workspace(const ScanDims& d) {   // (two column blocks: never zero, callers test for that)
  return std::max<size_t>(seg_layout(d, fwd_plan(d).nseg).total, blocks_of(d) == 2 ? 256 : 0);
}
size_t scan_tc_bwd_workspace(const ScanDims& d) {
  return std::max(scan_simt_bwd_workspace(d), tc_bwd_layout(d).total);
}
size_t scan_tc_states_bytes(const ScanDims& d) {   // two column blocks: one after the other
  return (size_t)d.batch * d.heads * chunks_of(d) * 64 * 128 * 2 * blocks_of(d);
}

int scan_tc_fwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                const float* z0, const void* Bprev, const void* Uprev, void* Y, float* zfinal,
                void* states_out, const ScanDims& d, int io_dtype, int y_dtype, void* ws, size_t ws_bytes,
                cudaStream_t st, const ScanLast* last) {
  SegPlan plan = fwd_plan(d);
  if (!ws || ws_bytes < scan_tc_fwd_workspace(d)) {   // N = 64 has always run without: the streams are then walked whole
    if (blocks_of(d) == 2) return SL_ERR_WORKSPACE_TOO_SMALL;
    plan = {1, chunks_of(d), 0, 0};
  }
  return scan_tc_fwd_impl(U, M, K, B, C, z0, Bprev, Uprev, Y, zfinal, states_out, d, plan,
                          reinterpret_cast<uint8_t*>(ws), io_dtype, y_dtype, st, last);
}

namespace {

// Tensor-core backward: state pre-sweep (unless the forward saved its chunk states), adjoint pre-pass when the
// sweep is split in time, reverse sweep, the boundary terms of carried B_prev / U_prev, and one launch for dM / dK from
// the scalars, the sum of the column blocks' dU (N = 128) and, for grouped B/C, that of dB / dC over the heads of a group.
template <typename TIn>
int run_bwd(const void* U, const float* M, const float* K, const void* B, const void* C, const float* z0,
            const void* Bprev, const void* Uprev, const void* states_in, const float* zfinal_in, const void* dY,
            const float* dfinal, void* dU, float* dM, float* dK, void* dB, void* dC, float* dinit, void* dBprev,
            void* dUprev, const ScanDims& d, int io_dtype, uint8_t* w, cudaStream_t st) {
  ensure_context();
  const TcBwdLayout lay = tc_bwd_layout(d);
  const bool bf = io_dtype == SL_BF16, grouped = d.groups != d.heads;
  const uint64_t BH = (uint64_t)d.batch * d.heads, BG = (uint64_t)d.batch * d.groups, W = 2 * (uint64_t)d.N;
  const int nC = chunks_of(d), nb = blocks_of(d);
  void* dBh = grouped ? (void*)(w + lay.dbh) : dB;   // where the sweep stores dB / dC (per head)
  void* dCh = grouped ? (void*)(w + lay.dch) : dC;
  const float* zfinal = zfinal_in;
  const void* states = states_in;
  if (!states || !zfinal) {   // nothing saved by the forward: recompute with the state pre-sweep
    float* zf = reinterpret_cast<float*>(w + lay.zfinal);
    if (int e = scan_tc_fwd_impl(U, M, K, B, nullptr, z0, Bprev, Uprev, nullptr, zf, w + lay.states, d, fwd_plan(d),
                                 w + lay.segs, io_dtype, SL_F32, st))
      return e;
    zfinal = zf;
    states = w + lay.states;
  }
  const SegPlan plan = bwd_plan(d);
  TcBwdParams p{};
  if (!tc::make_tmap_3d(&p.tmU, U, 64, d.T, BH, 64, bf) || !tc::make_tmap_3d(&p.tmB, B, W, d.T, BG, 64, bf) ||
      !tc::make_tmap_3d(&p.tmC, C, W, d.T, BG, 64, bf) || !tc::make_tmap_3d(&p.tmdY, dY, 64, d.T, BH, 64, bf) ||
      !tc::make_tmap_3d(&p.tmZ, states, 128, (uint64_t)nC * 64, BH * nb, 64, bf) ||
      !tc::make_tmap_3d(&p.tmdU[0], dU, 64, d.T, BH, 64, bf) ||
      (nb == 2 && !tc::make_tmap_3d(&p.tmdU[1], w + lay.du2, 64, d.T, BH, 64, bf)) ||
      !tc::make_tmap_3d(&p.tmdB, dBh, W, d.T, BH, 64, bf) || !tc::make_tmap_3d(&p.tmdC, dCh, W, d.T, BH, 64, bf))
    return SL_ERR_LAUNCH_FAILED;
  p.M = M; p.K = K; p.dfinal = dfinal; p.zfinal = zfinal;
  p.dg = reinterpret_cast<float2*>(w + lay.dg); p.sterm = reinterpret_cast<float2*>(w + lay.sterm);
  p.dkcd = reinterpret_cast<float2*>(w + lay.dkcd); p.anchor = reinterpret_cast<float2*>(w + lay.anchor);
  // with carried taps the adjoint of the start state is needed even when the caller asks for no d_initial
  float* dstart = dinit ? dinit : (Bprev ? reinterpret_cast<float*>(w + lay.dstart) : nullptr);
  float2* dgb = Bprev ? reinterpret_cast<float2*>(w + lay.dgb) : nullptr;
  p.dinit = dstart; p.T = d.T; p.N = d.N; p.nchunks = nC; p.cps = plan.cps; p.nseg = plan.nseg;
  p.tail = plan.tail; p.whole = plan.whole;
  p.heads = d.heads; p.groups = d.groups;
  p.wait_limit = wait_limit_clocks();
  if (plan.nseg > 1) {   // the adjoint at the end of every segment
    const SegLayout sl = seg_layout(d, plan.nseg);
    TcFwdParams q{};
    q.tmU = p.tmdY; q.tmB = p.tmC;
    q.M = M; q.K = K; q.heads = d.heads; q.groups = d.groups; q.T = d.T;
    q.nchunks = nC; q.cps = plan.cps; q.nseg = plan.nseg; q.wait_limit = p.wait_limit;
    q.tail = plan.tail; q.bh0 = plan.whole;
    q.seg = reinterpret_cast<float*>(w + lay.segs + sl.seg);
    q.seg_pi = reinterpret_cast<float2*>(w + lay.segs + sl.pi);
    if (int e = launch_prepass<TIn, 2>(q, (int)BH - plan.whole, nb, st)) return e;
    p.fold = plan.nseg <= FOLD_SEGS;
    if (!p.fold) {
      if (launch_chained(scan_tc_combine_kernel<TIn, true>, dim3((unsigned)BH, 16u * nb), 256, 0, st, true, q.seg, (const float2*)q.seg_pi,
                         dfinal, (const TIn*)nullptr, (const TIn*)nullptr, M, K, d.heads, d.groups, d.T, d.N, plan.nseg) != SL_OK)
        return SL_ERR_LAUNCH_FAILED;
      note_launches(1);
    }
    p.seg = q.seg; p.seg_pi = q.seg_pi;
  }
  {
    auto k = scan_tc_bwd_kernel<TIn, 4>;
    static std::atomic<unsigned long long> done{0};
    if (int e = ensure_smem(k, B_SMEM_BYTES, done)) return e;
    k<<<dim3((unsigned)BH, (unsigned)nb, (unsigned)plan.nseg), 576, B_SMEM_BYTES, st>>>(p);
    note_launches(1);
    if (int e = launch_status()) return e;
  }
  const TIn* bp = reinterpret_cast<const TIn*>(Bprev);
  if (Bprev) {
    scan_tc_bwd_boundary_kernel<TIn><<<(unsigned)BG, 256, 0, st>>>(
        dstart, bp, reinterpret_cast<const TIn*>(Uprev), M, K, reinterpret_cast<TIn*>(dBprev),
        reinterpret_cast<TIn*>(dUprev), dgb, d.heads, d.groups, d.T, d.N);
    note_launches(1);
  }
  TcPostParams q{};
  q.M = M; q.K = K; q.dg = p.dg; q.sterm = p.sterm; q.dkcd = p.dkcd; q.anchor = p.anchor; q.dg_boundary = dgb;
  q.dM = dM; q.dK = dK; q.dB = dB; q.dC = dC; q.dU = dU; q.dU2 = w + lay.du2;
  q.per_head_b = dBh; q.per_head_c = dCh;
  q.BH = (int)BH; q.heads = d.heads; q.groups = d.groups; q.T = d.T; q.nC = nC; q.D = (int)W;
  q.fin_blocks = (unsigned)(BH * ((nC + 3) / 4));
  q.red_blocks = grouped ? (unsigned)((BG * (size_t)d.T * (W / 8) + 127) / 128) : 0u;
  const unsigned add_blocks = nb == 2 ? (unsigned)((BH * (size_t)d.T * 8 + 127) / 128) : 0u;
  const unsigned blocks = q.fin_blocks + q.red_blocks + add_blocks;
  if (nb == 1) scan_tc_bwd_post_kernel<TIn, 1><<<blocks, 128, 0, st>>>(q);
  else scan_tc_bwd_post_kernel<TIn, 2><<<blocks, 128, 0, st>>>(q);
  note_launches(1);
  return launch_status();
}

}  // namespace

// A dY of another dtype than the operands (or none) takes the float32 sweeps.
int scan_tc_bwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                const float* z0, const void* Bprev, const void* Uprev, const void* states_in,
                const float* zfinal_in, const void* dY,
                const float* dfinal, void* dU, float* dM, float* dK, void* dB, void* dC, float* dinit,
                void* dBprev, void* dUprev, const ScanDims& d, int io_dtype, int dy_dtype, void* ws,
                size_t ws_bytes, cudaStream_t st) {
  if (!dY || dy_dtype != io_dtype)
    return scan_simt_bwd(U, M, K, B, C, z0, Bprev, Uprev, dY, dfinal, dU, dM, dK, dB, dC, dinit, dBprev,
                         dUprev, d, io_dtype, dy_dtype, ws, ws_bytes, st);
  if (!ws || ws_bytes < tc_bwd_layout(d).total) return SL_ERR_WORKSPACE_TOO_SMALL;
  uint8_t* w = reinterpret_cast<uint8_t*>(ws);
  return io_dtype == SL_BF16
             ? run_bwd<__nv_bfloat16>(U, M, K, B, C, z0, Bprev, Uprev, states_in, zfinal_in, dY, dfinal, dU, dM, dK, dB, dC,
                                      dinit, dBprev, dUprev, d, io_dtype, w, st)
             : run_bwd<__half>(U, M, K, B, C, z0, Bprev, Uprev, states_in, zfinal_in, dY, dfinal, dU, dM, dK, dB, dC, dinit,
                               dBprev, dUprev, d, io_dtype, w, st);
}

// The site code of the first expired wait on the current device since the last reset (0 = none).
int scan_tc_device_status(bool reset) {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int));
  if (reset && v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
  }
  return v;
}

}  // namespace sl
