// Shared device/host helpers for the slinoss_b200 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/slinoss_b200.h"

namespace sl {

// ---- element access in float32 -------------------------------------------------
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}
template <> __device__ __forceinline__ __half from_f32<__half>(float v) {
  // saturate to the finite range like the reference's output cast
  v = fminf(fmaxf(v, -65504.f), 65504.f);
  return __float2half_rn(v);
}

// Pairs: one packed conversion instead of two scalar ones.
template <typename T> __device__ __forceinline__ uint32_t pack_pair(float a, float b);
template <> __device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack_pair<__half>(float a, float b) {
  a = fminf(fmaxf(a, -65504.f), 65504.f); b = fminf(fmaxf(b, -65504.f), 65504.f);   // saturate like from_f32
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ float2 unpack_pair(uint32_t v);
template <> __device__ __forceinline__ float2 unpack_pair<__nv_bfloat16>(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 unpack_pair<__half>(uint32_t v) {
  return __half22float2(*reinterpret_cast<__half2*>(&v));
}
// a, b rounded to the io dtype and back (the roundings the reference makes between its steps)
template <typename T> __device__ __forceinline__ void round_pair(float& a, float& b) {
  if constexpr (sizeof(T) == 2) {
    const float2 r = unpack_pair<T>(pack_pair<T>(a, b));
    a = r.x; b = r.y;
  }
}

// 16-byte vectors of io elements: 4 floats or 8 16-bit values, handled as floats
template <typename T> struct Vec16 { static constexpr int N = 16 / (int)sizeof(T); };
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& r, float (&v)[Vec16<T>::N]);
template <typename T>
__device__ __forceinline__ void load16(const T* p, float (&v)[Vec16<T>::N]) {
  unpack16<T>(*reinterpret_cast<const uint4*>(p), v);
}
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& r, float (&v)[Vec16<T>::N]) {
  if constexpr (sizeof(T) == 2) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = unpack_pair<T>(w[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
  } else {
    v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
  }
}
template <typename T>
__device__ __forceinline__ void store16(T* p, const float (&v)[Vec16<T>::N]) {
  if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_pair<T>(v[0], v[1]), pack_pair<T>(v[2], v[3]),
                                              pack_pair<T>(v[4], v[5]), pack_pair<T>(v[6], v[7]));
  } else {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

struct cf {  // complex float
  float re, im;
};
__device__ __forceinline__ cf cmul(cf a, cf b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cf cmul_conj_a(cf a, cf b) {  // conj(a) * b
  return {a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re};
}
__device__ __forceinline__ cf cadd(cf a, cf b) { return {a.re + b.re, a.im + b.im}; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- packed float32 pairs (two independent lanes per instruction) ---------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 mk2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 dup2(float v) { return mk2(v, v); }
__device__ __forceinline__ float2 un2(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// 2^x, log2(x) and 1/x on the special-function unit
__device__ __forceinline__ float ex2f(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float lg2f(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcpf(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// (1 ulp for the reciprocal, and 0 for a denominator beyond 2^126, which is the right limit here)
__device__ __forceinline__ float sigmoid_f(float x) { return rcpf(1.f + ex2f(-1.4426950408889634f * x)); }
__device__ __forceinline__ float silu_f(float x) { return x * sigmoid_f(x); }
__device__ __forceinline__ f2 sigmoid2(f2 x) {
  const float2 e = un2(mul2(x, dup2(-1.4426950408889634f)));
  const float2 d = un2(add2(mk2(ex2f(e.x), ex2f(e.y)), dup2(1.f)));
  return mk2(rcpf(d.x), rcpf(d.y));
}

// 16-bit rows take the one-instruction tanh (relative error 2^-11, below the rounding of the output);
// float32 rows the precise one.
template <bool FAST> __device__ __forceinline__ float tanh_io(float x) {
  if (FAST) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  }
  return tanhf(x);
}
template <bool FAST> __device__ __forceinline__ float gelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.f + tanh_io<FAST>(u));
}

// d += a b on the tensor cores: 16 rows by 8 columns, 16 values of k
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
// 16 bytes to shared memory; of ``bytes`` of them that are read the rest is zeroed
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// ---- chains of launches ----------------------------------------------------------
// A kernel launched as dependent may start while its predecessor in the stream still runs; it does what needs nothing of the
// predecessor (its weights) and then waits for the end of that grid.  Every kernel that such a launch may follow releases it at its start.
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- host side -----------------------------------------------------------------
// remembers the CUDA error behind the last SL_ERR_LAUNCH_FAILED (see sl_last_cuda_error)
void note_cuda_error(int code);

template <typename K, typename A, typename... As>
inline int launch_chained(K kernel, dim3 grid, unsigned block, size_t smem, cudaStream_t st, bool dependent, const A& a,
                          const As&... as) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cfg.attrs = &attr; cfg.numAttrs = dependent ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a, as...);
  if (e == cudaSuccess) return SL_OK;
  cudaGetLastError();
  note_cuda_error((int)e);
  return SL_ERR_LAUNCH_FAILED;
}

inline size_t dtype_size(int dt) { return dt == SL_F32 ? 4 : 2; }
inline bool dtype_ok(int dt) { return dt == SL_F32 || dt == SL_BF16 || dt == SL_F16; }
inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// process-wide count of kernels this library has launched (see sl_kernel_launches)
void note_launches(int n);

inline int launch_status() {
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return SL_OK;
  note_cuda_error((int)e);
  return SL_ERR_LAUNCH_FAILED;
}

// Kernel attributes stick to a device: set once per (kernel, device) instead of on every launch.
template <typename F>
inline int ensure_smem(F k, size_t bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SL_ERR_LAUNCH_FAILED;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_relaxed) & bit) return SL_OK;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return SL_ERR_LAUNCH_FAILED;
  done.fetch_or(bit, std::memory_order_relaxed);
  return SL_OK;
}

// Dispatch a callable templated on the io element type.
#define SL_DISPATCH_DTYPE(dt, T, ...)                         \
  do {                                                        \
    if ((dt) == SL_F32) {                                     \
      using T = float;                                        \
      __VA_ARGS__;                                            \
    } else if ((dt) == SL_BF16) {                             \
      using T = __nv_bfloat16;                                \
      __VA_ARGS__;                                            \
    } else {                                                  \
      using T = __half;                                       \
      __VA_ARGS__;                                            \
    }                                                         \
  } while (0)

// ---- internal entry points implemented in the other translation units ----------
struct ScanDims {
  int batch, heads, groups, T, P, N, chunk;
};

int scan_simt_fwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                  const float* z0, const void* Bprev, const void* Uprev, void* Y, float* zfinal,
                  const ScanDims& d, int io_dtype, int y_dtype, void* ws, size_t ws_bytes, cudaStream_t st);
size_t scan_simt_fwd_workspace(const ScanDims& d);
size_t scan_simt_bwd_workspace(const ScanDims& d);
size_t scan_simt_bwd_split_workspace(const ScanDims& d);
int scan_simt_bwd(const void* U, const float* M, const float* K, const void* B, const void* C,
                  const float* z0, const void* Bprev, const void* Uprev, const void* dY,
                  const float* dfinal, void* dU, float* dM, float* dK, void* dB, void* dC,
                  float* dinit, void* dBprev, void* dUprev, const ScanDims& d, int io_dtype,
                  int dy_dtype, void* ws, size_t ws_bytes, cudaStream_t st);
bool scan_simt_supported(const ScanDims& d);

}  // namespace sl
