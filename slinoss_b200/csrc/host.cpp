// Host module of the package: the launchers of the C ABI for torch tensors, in native code.
//
// A launch from Python cost 15 to 30 us of interpreter time (argument conversion of up to 40 ctypes arguments, device
// guard, stream lookup, output allocation); the same work takes 2 to 4 us here.  Every function allocates its outputs
// and scratch with torch, launches on torch's current stream and turns status codes into exceptions.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/as_strided_native.h>
#include <ATen/ops/mm_cuda_dispatch.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <cmath>

#include "../../include/slinoss_b200.h"
#include "host_abi.h"

namespace py = pybind11;

namespace {

using at::Tensor;
using OptT = c10::optional<Tensor>;

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SL_F32;
    case at::kBFloat16: return SL_BF16;
    case at::kHalf: return SL_F16;
    default: throw pybind11::value_error("unsupported dtype; expected float32, bfloat16 or float16");
  }
}
at::ScalarType type_of(int code) { return code == SL_F32 ? at::kFloat : code == SL_BF16 ? at::kBFloat16 : at::kHalf; }

void check(int status, const char* what) {
  if (status == SL_OK) return;
  std::string text = std::string("slinoss_b200.") + what + " failed with status " + std::to_string(status) + ": " +
                     sl_status_string(status);
  if (status == SL_ERR_LAUNCH_FAILED) text += std::string(" (") + sl_last_cuda_error() + ")";
  throw std::runtime_error(text);
}

// Device guard and stream of a call; every tensor handed to it must live on one CUDA device.
struct Call {
  c10::cuda::OptionalCUDAGuard guard;
  c10::Device dev{c10::kCPU};
  bool any = false;
  void need(const Tensor& t) {
    if (!t.is_cuda()) throw pybind11::value_error("slinoss_b200 kernels require CUDA tensors.");
    if (!any) { dev = t.device(); any = true; }
    else if (t.device() != dev) throw pybind11::value_error("All tensors must be on the same device.");
  }
  void need(const OptT& t) { if (t) need(*t); }
  template <typename... Ts> explicit Call(const Ts&... ts) { (need(ts), ...); guard.set_device(dev); }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
  Tensor empty(at::IntArrayRef shape, at::ScalarType t) const { return at::empty(shape, at::TensorOptions().dtype(t).device(dev)); }
  Tensor zeros(at::IntArrayRef shape, at::ScalarType t) const { return at::zeros(shape, at::TensorOptions().dtype(t).device(dev)); }
  Tensor bytes(size_t n) const { return empty({(int64_t)n}, at::kByte); }
};

const void* ptr(const Tensor& t) { return t.data_ptr(); }
const void* ptr(const OptT& t) { return t ? t->data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.data_ptr(); }
void* mptr(const OptT& t) { return t ? t->data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return static_cast<const float*>(t.data_ptr()); }
const float* fptr(const OptT& t) { return t ? static_cast<const float*>(t->data_ptr()) : nullptr; }
float* mfptr(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
float* mfptr(const OptT& t) { return t ? static_cast<float*>(t->data_ptr()) : nullptr; }

uint8_t* column(const Tensor& rows, int64_t c) { return static_cast<uint8_t*>(rows.data_ptr()) + c * rows.element_size(); }

using Config = std::array<float, 10>;
sl_scanprep_config config_of(const Config& c) {
  return sl_scanprep_config{c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9]};
}

// ---- scan ---------------------------------------------------------------------------------------------------------
std::tuple<Tensor, OptT, OptT> scan_fwd(const Tensor& U, const Tensor& M, const Tensor& K, const Tensor& B, const Tensor& C,
                                        const OptT& z0, const OptT& Bp, const OptT& Up, int chunk, int y_code,
                                        bool want_final, int path, bool save_states) {
  Call call(U, M, K, B, C, z0, Bp, Up);
  const int batch = U.size(0), heads = U.size(1), T = U.size(2), P = U.size(3), groups = B.size(1), N = B.size(3) / 2;
  const int io = code_of(U.scalar_type());
  Tensor Y = call.empty({batch, heads, T, P}, type_of(y_code));
  OptT final_state, states, ws;
  if (save_states) {
    const size_t n = sl_workspace_bytes(SL_WS_SCAN_STATES, batch, heads, groups, T, P, N, chunk, io, path);
    if (n) states = call.bytes(n);
  }
  if (want_final || states) final_state = call.empty({batch, heads, P, 2 * N}, at::kFloat);
  const size_t n = sl_workspace_bytes(SL_WS_SCAN_FWD, batch, heads, groups, T, P, N, chunk, io, path);
  if (n) ws = call.bytes(n);
  check(sl_v2x2ssd_fwd(ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), fptr(z0), ptr(Bp), ptr(Up), mptr(Y), mfptr(final_state),
                       mptr(states), batch, heads, groups, T, P, N, chunk, io, y_code, path, mptr(ws), n, call.stream()),
        "sl_v2x2ssd_fwd");
  return {Y, final_state, states};
}

// the same with the end state and the last rows of B and U, all in the type of the operands; nothing where the tensor-core path
// does not run
c10::optional<std::tuple<Tensor, Tensor, Tensor, Tensor>> scan_fwd_last(const Tensor& U, const Tensor& M, const Tensor& K,
                                                                        const Tensor& B, const Tensor& C, const OptT& z0, const OptT& Bp,
                                                                        const OptT& Up, int chunk, int path) {
  Call call(U, M, K, B, C, z0, Bp, Up);
  const int batch = U.size(0), heads = U.size(1), T = U.size(2), P = U.size(3), groups = B.size(1), N = B.size(3) / 2;
  const auto type = U.scalar_type();
  if ((type != at::kBFloat16 && type != at::kHalf) || P != 64 || (N != 64 && N != 128) || path == SL_PATH_SIMT) return {};
  const int io = code_of(type);
  Tensor Y = call.empty({batch, heads, T, P}, type), state = call.empty({batch, heads, P, 2 * N}, type);
  Tensor B_last = call.empty({batch, groups, 2 * N}, type), U_last = call.empty({batch, heads, P}, type);
  const size_t n = sl_workspace_bytes(SL_WS_SCAN_FWD, batch, heads, groups, T, P, N, chunk, io, path);
  OptT ws;
  if (n) ws = call.bytes(n);
  const int rc = sl::scan_fwd_last(ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), fptr(z0), ptr(Bp), ptr(Up), mptr(Y),
                                   sl::ScanLast{mptr(state), mptr(B_last), mptr(U_last)}, batch, heads, groups, T, P, N, chunk, io, path,
                                   mptr(ws), n, call.stream());
  if (rc == SL_ERR_UNSUPPORTED) return {};
  check(rc, "sl_v2x2ssd_fwd");
  return std::make_tuple(Y, state, B_last, U_last);
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, OptT, OptT, OptT> scan_bwd(
    const Tensor& U, const Tensor& M, const Tensor& K, const Tensor& B, const Tensor& C, const OptT& z0, const OptT& Bp,
    const OptT& Up, const OptT& states, const OptT& final_state, const OptT& dY, const OptT& dfinal, int chunk, int path) {
  Call call(U, M, K, B, C, z0, Bp, Up, dY, dfinal);
  const int batch = U.size(0), heads = U.size(1), T = U.size(2), P = U.size(3), groups = B.size(1), N = B.size(3) / 2;
  const int io = code_of(U.scalar_type()), dy = dY ? code_of(dY->scalar_type()) : io;
  Tensor dU = at::empty_like(U), dM = call.empty({batch, heads, T, 2}, at::kFloat);
  Tensor dK = call.empty({batch, heads, T, 2, 2}, at::kFloat), dB = at::empty_like(B), dC = at::empty_like(C);
  OptT dinit, dBp, dUp, ws;
  if (z0) dinit = call.empty({batch, heads, P, 2 * N}, at::kFloat);
  if (Bp) dBp = at::empty_like(*Bp);
  if (Up) dUp = at::empty_like(*Up);
  const size_t n = sl_workspace_bytes(SL_WS_SCAN_BWD, batch, heads, groups, T, P, N, chunk, io, path);
  if (n) ws = call.bytes(n);
  check(sl_v2x2ssd_bwd(ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), fptr(z0), ptr(Bp), ptr(Up), ptr(states), fptr(final_state),
                       ptr(dY), fptr(dfinal), mptr(dU), mfptr(dM), mfptr(dK), mptr(dB), mptr(dC), mfptr(dinit), mptr(dBp),
                       mptr(dUp), batch, heads, groups, T, P, N, chunk, io, dy, path, mptr(ws), n, call.stream()),
        "sl_v2x2ssd_bwd");
  return {dU, dM, dK, dB, dC, dinit, dBp, dUp};
}

std::tuple<Tensor, Tensor> scan_decode(const Tensor& U, const Tensor& M, const Tensor& K, const Tensor& B, const Tensor& C,
                                       const Tensor& state, const OptT& Bp, const OptT& Up, int y_code, const OptT& state_out) {
  Call call(U, M, K, B, C, state, Bp, Up);
  const int batch = U.size(0), heads = U.size(1), P = U.size(2), groups = B.size(1), N = B.size(2) / 2;
  Tensor Y = call.empty({batch, heads, P}, type_of(y_code));
  Tensor out = state_out ? *state_out : at::empty_like(state);
  check(sl_v2x2ssd_decode(ptr(U), fptr(M), fptr(K), ptr(B), ptr(C), fptr(state), ptr(Bp), ptr(Up), mptr(Y), mfptr(out), batch,
                          heads, groups, P, N, code_of(U.scalar_type()), y_code, call.stream()),
        "sl_v2x2ssd_decode");
  return {Y, out};
}

// ---- scan preparation (+ causal conv) -------------------------------------------------------------------------------
// (batch, T, C) rows in a layout with dense channels and batch stride T * row stride, copied only if needed
Tensor as_rows(const Tensor& x) {
  if (x.stride(2) == 1 && (x.size(0) == 1 || x.stride(0) == x.size(1) * x.stride(1)) &&
      (x.size(1) > 1 || x.stride(1) >= x.size(2)))
    return x;
  return x.contiguous();
}
int64_t row_stride(const Tensor& x) { return x.size(1) > 1 ? x.stride(1) : std::max<int64_t>(x.stride(1), x.size(2)); }

struct ULayout { int64_t b = 0, h = 0, t = 0; };
ULayout u_layout(bool bhtp, int64_t heads, int64_t T, int64_t P) {
  return bhtp ? ULayout{heads * T * P, T * P, P} : ULayout{T * heads * P, P, heads * P};
}
struct Biases { const float* p[5] = {nullptr, nullptr, nullptr, nullptr, nullptr}; };
Biases biases_of(const std::vector<Tensor>& v) {
  Biases b;
  for (size_t i = 0; i < v.size() && i < 5; ++i) b.p[i] = fptr(v[i]);
  return b;
}

std::tuple<OptT, OptT, OptT, OptT, OptT, OptT> scanprep_fwd(const OptT& value, const OptT& w, const OptT& bias, const OptT& st,
                                                            const OptT& params, const OptT& bc,
                                                            const std::vector<Tensor>& biases, const c10::optional<Config>& cfg,
                                                            int heads, int P, bool bhtp, bool want_state) {
  const Tensor& ref = value ? *value : params ? *params : *bc;
  Call call(value, w, bias, st, params, bc);
  for (const auto& t : biases) call.need(t);
  const int64_t batch = ref.size(0), T = ref.size(1);
  OptT U, M, K, Bo, Co, nstate, rows;
  ULayout lay;
  int64_t vstride = 0;
  int d_conv = 1, groups = 1, N = 1;
  if (value) {
    rows = as_rows(*value);
    vstride = row_stride(*rows);
    lay = u_layout(bhtp, heads, T, P);
    U = bhtp ? call.empty({batch, heads, T, P}, value->scalar_type()) : call.empty({batch, T, (int64_t)heads * P}, value->scalar_type());
    if (w) {
      d_conv = w->size(1);
      if (want_state) nstate = call.empty({batch, (int64_t)heads * P, d_conv - 1}, value->scalar_type());
    }
  }
  if (bc) {
    groups = bc->size(2); N = bc->size(4);
    Bo = call.empty({batch, groups, T, 2 * N}, bc->scalar_type());
    Co = call.empty({batch, groups, T, 2 * N}, bc->scalar_type());
  }
  if (params) {
    M = call.empty({batch, heads, T, 2}, at::kFloat);
    K = call.empty({batch, heads, T, 2, 2}, at::kFloat);
  }
  const Biases bs = biases_of(biases);
  sl_scanprep_config c{};
  if (cfg) c = config_of(*cfg);
  check(sl_scanprep_conv_fwd(ptr(rows), vstride, ptr(w), ptr(bias), ptr(st), mptr(nstate), d_conv, ptr(params), ptr(bc), bs.p[0],
                             bs.p[1], bs.p[2], bs.p[3], bs.p[4], cfg ? &c : nullptr, mptr(U), lay.b, lay.h, lay.t, mfptr(M),
                             mfptr(K), mptr(Bo), mptr(Co), batch, heads, groups, T, P, N, code_of(ref.scalar_type()),
                             call.stream()),
        "sl_scanprep_conv_fwd");
  return {U, M, K, Bo, Co, nstate};
}

// d_value | d_conv_weight | d_conv_bias | d_conv_state | d_params | d_bc | d_dt_bias | d_alpha_bias | d_theta_mod_bias |
// d_theta_bias.  The float32 accumulators are slices of one zeroed buffer.
std::vector<OptT> scanprep_bwd(const OptT& value, const OptT& w, const OptT& bias, const OptT& st, const OptT& params,
                               const OptT& bc, const std::vector<Tensor>& biases, const c10::optional<Config>& cfg,
                               const OptT& dU, const OptT& dM, const OptT& dK, const OptT& dBo, const OptT& dCo, int heads,
                               int P, bool bhtp, bool want_dstate) {
  const Tensor& ref = value ? *value : params ? *params : *bc;
  Call call(value, w, bias, st, params, bc, dU, dM, dK, dBo, dCo);
  const int64_t batch = ref.size(0), T = ref.size(1), C = (int64_t)heads * P;
  std::vector<OptT> out(10);
  ULayout lay;
  int64_t vstride = 0;
  int d_conv = w ? w->size(1) : 1, groups = 1, N = 1;
  OptT rows, gU, gM, gK, gB, gC;
  const int64_t nw = dU && w ? C * d_conv : 0, nb = dU && w ? C : 0, nh = dM ? 4 * heads : 0;
  Tensor acc;
  if (nw + nb + nh) acc = call.zeros({nw + nb + nh}, at::kFloat);
  if (dU) {
    rows = as_rows(*value);
    vstride = row_stride(*rows);
    gU = dU->contiguous();
    lay = u_layout(bhtp, heads, T, P);
    out[0] = call.empty({batch, T, C}, value->scalar_type());
    if (w) {
      out[1] = acc.narrow(0, 0, nw).view({C, d_conv});
      out[2] = acc.narrow(0, nw, nb);
      if (want_dstate && d_conv > 1) out[3] = call.zeros({batch, C, d_conv - 1}, value->scalar_type());
    }
  }
  if (dBo) {
    groups = bc->size(2); N = bc->size(4);
    gB = dBo->contiguous(); gC = dCo->contiguous();
    out[5] = call.empty(bc->sizes(), bc->scalar_type());
  }
  if (dM) {
    gM = dM->contiguous(); gK = dK->contiguous();
    out[4] = call.empty(params->sizes(), params->scalar_type());
    for (int i = 0; i < 4; ++i) out[6 + i] = acc.narrow(0, nw + nb + i * heads, heads);
  }
  const Biases bs = biases_of(biases);
  sl_scanprep_config c{};
  if (cfg) c = config_of(*cfg);
  check(sl_scanprep_conv_bwd(ptr(rows), vstride, ptr(w), ptr(bias), ptr(st), d_conv, ptr(params), ptr(bc), bs.p[0], bs.p[1],
                             bs.p[2], bs.p[3], bs.p[4], cfg ? &c : nullptr, ptr(gU), lay.b, lay.h, lay.t, fptr(gM), fptr(gK),
                             ptr(gB), ptr(gC), mptr(out[0]), mfptr(out[1]), mfptr(out[2]), mptr(out[3]), mptr(out[4]),
                             mptr(out[5]), mfptr(out[6]), mfptr(out[7]), mfptr(out[8]), mfptr(out[9]), batch, heads, groups, T,
                             P, N, code_of(ref.scalar_type()), call.stream()),
        "sl_scanprep_conv_bwd");
  return out;
}

// ---- mixer tail, RMSNorm, FFN activation --------------------------------------------------------------------------------
Tensor tail_fwd(const Tensor& Y, const Tensor& gate_in, const OptT& skip, const OptT& d_skip, const Tensor& w, float eps) {
  Call call(Y, gate_in, skip, d_skip, w);
  const Tensor gate = as_rows(gate_in);
  const int64_t batch = Y.size(0), heads = Y.size(1), T = Y.size(2), P = Y.size(3);
  Tensor normed = call.empty({batch, T, heads * P}, Y.scalar_type());
  check(sl_mixer_tail_fwd(ptr(Y), ptr(gate), row_stride(gate), ptr(skip), fptr(d_skip), ptr(w), eps, mptr(normed), batch, heads,
                          T, P, code_of(Y.scalar_type()), call.stream()),
        "sl_mixer_tail_fwd");
  return normed;
}

std::tuple<Tensor, Tensor, OptT, OptT, Tensor> tail_bwd(const Tensor& Y, const Tensor& gate_in, const OptT& skip,
                                                        const OptT& d_skip, const Tensor& w, float eps, const Tensor& dn_in) {
  Call call(Y, gate_in, skip, d_skip, w, dn_in);
  const Tensor gate = as_rows(gate_in), dn = dn_in.contiguous();
  const int64_t batch = Y.size(0), heads = Y.size(1), T = Y.size(2), P = Y.size(3), nh = skip ? heads : 0;
  Tensor dY = at::empty_like(Y), dgate = call.empty({batch, T, heads * P}, Y.scalar_type());
  Tensor acc = call.zeros({heads * P + nh}, at::kFloat), dw = acc.narrow(0, 0, heads * P);
  OptT dskip_in, dd;
  if (skip) { dskip_in = at::empty_like(Y); dd = acc.narrow(0, heads * P, nh); }
  check(sl_mixer_tail_bwd(ptr(Y), ptr(gate), row_stride(gate), ptr(skip), fptr(d_skip), ptr(w), eps, ptr(dn), mptr(dY), mptr(dgate),
                          mptr(dskip_in), mfptr(dd), mfptr(dw), batch, heads, T, P, code_of(Y.scalar_type()), call.stream()),
        "sl_mixer_tail_bwd");
  return {dY, dgate, dskip_in, dd, dw};
}

Tensor rmsnorm_fwd(const Tensor& x, const Tensor& w, float eps) {
  Call call(x, w);
  const int64_t C = x.size(-1);
  Tensor out = at::empty_like(x);
  check(sl_rmsnorm_fwd(ptr(x), ptr(w), eps, mptr(out), x.numel() / C, C, code_of(x.scalar_type()), call.stream()), "sl_rmsnorm_fwd");
  return out;
}
// ``extra`` is added to dx
std::tuple<Tensor, Tensor> rmsnorm_bwd(const Tensor& x, const Tensor& w, float eps, const Tensor& dy, const OptT& extra, bool as_rows_type) {
  Call call(x, w, dy, extra);
  const int64_t C = x.size(-1);
  Tensor dx = at::empty_like(x), dw = call.zeros({C}, at::kDouble);
  check(sl::rmsnorm_bwd(ptr(x), ptr(w), eps, ptr(dy), ptr(extra), mptr(dx), nullptr, dw.data_ptr<double>(), nullptr, x.numel() / C, C,
                        code_of(x.scalar_type()), static_cast<cudaStream_t>(call.stream())),
        "sl_rmsnorm_bwd");
  return {dx, dw.to(as_rows_type ? x.scalar_type() : at::kFloat)};
}
Tensor column_sum(const Tensor& x) {
  Call call(x);
  const int64_t C = x.size(-1), rows = x.numel() / C;
  const int io = code_of(x.scalar_type());
  Tensor out = call.empty({C}, x.scalar_type());
  const Tensor partial = call.empty({(int64_t)sl::column_sum_partials(rows, C, io)}, at::kFloat);
  check(sl::column_sum(ptr(x), mptr(out), mfptr(partial), rows, C, io, static_cast<cudaStream_t>(call.stream())), "column_sum");
  return out;
}
Tensor ffn_act_fwd(const Tensor& proj, int kind) {
  Call call(proj);
  const int64_t W = proj.size(-1), H = kind == 1 ? W / 2 : W;
  auto shape = proj.sizes().vec();
  shape.back() = H;
  Tensor hidden = call.empty(shape, proj.scalar_type());
  check(sl_ffn_activation_fwd(ptr(proj), mptr(hidden), proj.numel() / W, H, kind, code_of(proj.scalar_type()), call.stream()),
        "sl_ffn_activation_fwd");
  return hidden;
}
Tensor ffn_act_bwd(const Tensor& proj, const Tensor& dhid, int kind) {
  Call call(proj, dhid);
  const int64_t W = proj.size(-1), H = kind == 1 ? W / 2 : W;
  Tensor dproj = at::empty_like(proj);
  check(sl_ffn_activation_bwd(ptr(proj), ptr(dhid), mptr(dproj), proj.numel() / W, H, kind, code_of(proj.scalar_type()), call.stream()),
        "sl_ffn_activation_bwd");
  return dproj;
}

// ---- decode: one token of a mixer ------------------------------------------------------------------------------------
// y = W x: the small-batch kernel where it applies, else the library GEMM, which also says what is wrong with operands that
// do not fit together.
bool small_batch(at::ScalarType type, int64_t rows, int64_t K, const Tensor& W, const OptT& bias) {
  return rows <= 64 && K % 8 == 0 && K <= 4096 && type != at::kFloat && W.scalar_type() == type && W.dim() == 2 && W.size(1) == K &&
         W.is_contiguous() && (!bias || (bias->scalar_type() == type && bias->is_contiguous() && bias->numel() == W.size(0)));
}
bool small_batch(const Tensor& x, const Tensor& W, const OptT& bias) {
  return small_batch(x.scalar_type(), x.size(0), x.size(1), W, bias) && x.stride(1) == 1 && x.stride(0) % 8 == 0;
}
Tensor linear_rows(const Call& call, const Tensor& x, const Tensor& W, const OptT& bias, const OptT& out_in) {
  const int64_t M = x.size(0), K = x.size(1), O = W.size(0);
  if (small_batch(x, W, bias)) {
    Tensor out = out_in ? *out_in : call.empty({M, O}, x.scalar_type());
    const sl::SkinnyArgs a{ptr(x), x.stride(0), nullptr, 0.f, nullptr, 0, ptr(W), ptr(bias), mptr(out), (int)M, (int)K, (int)O,
                           code_of(x.scalar_type())};
    check(sl::skinny_linear(a, static_cast<cudaStream_t>(call.stream())), "skinny_linear");
    return out;
  }
  if (out_in && !bias) { Tensor y = *out_in; at::mm_out(y, x, W.t()); return y; }
  const Tensor y = at::linear(x, W, bias);
  if (out_in) { out_in->copy_(y); return *out_in; }
  return y;
}

// One token x (batch, d_model) -> mixer(x).  conv, state and u_prev are updated in place; the new b_prev goes to b_prev
// itself when every head has its own group, else to a tensor of its own (the heads of a group read the old one at different
// times).
std::tuple<Tensor, Tensor, Tensor> mixer_token(const Tensor& x, const Tensor& in_w, const Tensor& dw_w, const Tensor& dw_b,
                                               const std::vector<Tensor>& biases, const Config& cfg, const Tensor& d_skip,
                                               const Tensor& norm_w, float norm_eps, const Tensor& out_w, const OptT& out_b,
                                               const Tensor& conv, const Tensor& state, const Tensor& b_prev,
                                               const Tensor& u_prev, const OptT& workspace, int heads, int groups, int P, int N,
                                               const OptT& out) {
  Call call(x, in_w, dw_w, dw_b, d_skip, norm_w, out_w, out_b, conv, state, b_prev, u_prev, workspace, out);
  for (const auto& t : biases) call.need(t);
  const int64_t batch = x.size(0), C = (int64_t)heads * P, O = in_w.size(0);
  const int io = code_of(x.scalar_type());
  if (O != 2 * C + 3 * heads + 4 * (int64_t)groups * N) throw pybind11::value_error("in_proj does not fit the mixer's sizes.");
  for (const Tensor& t : {conv, b_prev, u_prev})
    if (t.scalar_type() != x.scalar_type()) throw pybind11::value_error("the decode state does not have the token's type.");
  const bool chained = small_batch(x, in_w, {});   // the step may start behind our own in_proj kernel
  const Tensor proj = linear_rows(call, x, in_w, {}, {});
  const size_t ws_bytes = sl_mixer_decode_step_workspace_bytes(batch, heads, P);
  Tensor ws = workspace && (size_t)workspace->numel() >= ws_bytes ? *workspace : call.bytes(ws_bytes);
  Tensor b_next = groups == heads ? b_prev : at::empty_like(b_prev);
  const Biases bs = biases_of(biases);
  const sl_scanprep_config c = config_of(cfg);
  const auto* base = static_cast<const uint8_t*>(proj.data_ptr());
  const int64_t e = proj.element_size();
  const sl::MixerStepArgs a{base, base + C * e, base + 2 * C * e, base + (2 * C + 3 * heads) * e, O, O, O, O, ptr(dw_w), ptr(dw_b),
                            mptr(conv), (int)dw_w.size(1), bs.p[0], bs.p[1], bs.p[2], bs.p[3], bs.p[4], &c, fptr(d_skip),
                            mfptr(state), ptr(b_prev), mptr(b_next), mptr(u_prev), mptr(ws), (size_t)ws.numel(), (int)batch, heads,
                            groups, P, N, io, chained};
  const auto st = static_cast<cudaStream_t>(call.stream());
  check(sl::mixer_step_launch(a, st), "mixer_step");
  const int64_t K = C, OO = out_w.size(0);
  if (small_batch(x.scalar_type(), batch, K, out_w, out_b)) {   // the row norm inside the projection
    Tensor y = out ? *out : call.empty({batch, OO}, x.scalar_type());
    const sl::SkinnyArgs s{mptr(ws), C, ptr(norm_w), norm_eps, sl::step_partials(mptr(ws), batch, heads, P), 8 * heads, ptr(out_w),
                           ptr(out_b), mptr(y), (int)batch, (int)K, (int)OO, io, true};
    check(sl::skinny_linear(s, st), "skinny_linear");
    return {y, b_next, ws};
  }
  Tensor normed = call.empty({batch, C}, x.scalar_type());
  check(sl::mixer_step_norm(mptr(ws), ptr(norm_w), norm_eps, mptr(normed), batch, heads, P, io, st), "mixer_step");
  return {linear_rows(call, normed, out_w, out_b, out), b_next, ws};
}

// One token of a mixer, or of a whole block, without Python per launch.  A plan holds the parameters of one module (the
// tensors themselves, so data that moves or changes type is seen) and a list of guards: dictionary entries that must still be
// the objects they were or still be absent, and dictionaries that must still be empty (hooks).  Checking the guards costs 2 us, what
// they replace - attribute lookups, conversions of 30 arguments, checks of every tensor - cost 25 us per block.
//
// The module keeps its plan in its own __dict__, so the plan does not hold that one: its entries are guards without a
// dictionary, and valid() is given it.  What the plan does hold it shows to the garbage collector, for modules that lie on a
// cycle of the program's own.
class TokenPlan {
 public:
  // same: (dict or None for the module's own, key[, object]), without an object: no such entry;
  // params: in_w dw_w dw_b dt alpha theta_mod theta theta_sign d_skip norm_w out_w out_b; branch: pre_norm [ffn_norm w1 b1 w2 b2]
  TokenPlan(std::vector<py::tuple> same, std::vector<py::dict> empty, std::vector<OptT> params, std::vector<OptT> branch,
            std::vector<double> eps, const Config& cfg, std::array<int64_t, 5> dims, int ffn_kind)
      : same_(std::move(same)), empty_(std::move(empty)), p_(std::move(params)), b_(std::move(branch)), eps_(std::move(eps)),
        cfg_(config_of(cfg)), heads_(dims[0]), groups_(dims[1]), P_(dims[2]), N_(dims[3]), d_conv_(dims[4]), ffn_kind_(ffn_kind) {
    if (p_.size() != 12 || (b_.size() != 0 && b_.size() != 1 && b_.size() != 6) || eps_.size() != 3)
      throw pybind11::value_error("bad plan.");
  }

  bool valid(const py::dict& own) const {
    if (cleared_) return false;
    for (const auto& g : same_) {
      PyObject* const d = PyTuple_GET_ITEM(g.ptr(), 0);
      PyObject* const want = PyTuple_GET_SIZE(g.ptr()) == 3 ? PyTuple_GET_ITEM(g.ptr(), 2) : nullptr;
      if (PyDict_GetItem(d == Py_None ? own.ptr() : d, PyTuple_GET_ITEM(g.ptr(), 1)) != want) return false;
    }
    for (const auto& d : empty_)
      if (PyDict_Size(d.ptr()) != 0) return false;
    return true;
  }

  static void collectable(PyHeapTypeObject* heap) {
    PyTypeObject* const type = &heap->ht_type;
    type->tp_flags |= Py_TPFLAGS_HAVE_GC;
    type->tp_traverse = [](PyObject* self, visitproc visit, void* arg) {
      Py_VISIT(Py_TYPE(self));
      if (const TokenPlan* const plan = of(self)) {
        for (const auto& g : plan->same_) Py_VISIT(g.ptr());
        for (const auto& d : plan->empty_) Py_VISIT(d.ptr());
      }
      return 0;
    };
    type->tp_clear = [](PyObject* self) {
      if (TokenPlan* const plan = of(self)) {
        plan->cleared_ = true;
        plan->same_.clear(); plan->empty_.clear(); plan->p_.clear(); plan->b_.clear();
      }
      return 0;
    };
  }

  // None where the call is not the plain one; else (out, next b_prev, workspace).  behind_own: nothing was queued since another
  // plan's token left its last kernel on this stream.
  py::object step(const Tensor& x, const OptT& conv, const OptT& state, const OptT& b_prev, const OptT& u_prev,
                  const OptT& workspace, bool behind_own) const {
    if (cleared_ || at::GradMode::is_enabled() || at::autocast::is_autocast_enabled(at::kCUDA) || !x.is_cuda() || x.dim() != 2)
      return py::none();
    const auto type = x.scalar_type();
    const int64_t M = x.size(0), D = x.size(1), C = heads_ * P_;
    if ((type != at::kBFloat16 && type != at::kHalf) || M < 1) return py::none();
    auto is = [&](const OptT& t, at::ScalarType ty, at::IntArrayRef shape) {
      return t && t->scalar_type() == ty && t->device() == x.device() && t->is_contiguous() && t->sizes() == shape;
    };
    const int64_t O = 2 * C + 3 * heads_ + 4 * groups_ * N_;
    bool ok = is(p_[0], type, {O, D}) && is(p_[1], type, {C, d_conv_}) && is(p_[2], type, {C}) && is(p_[9], type, {C}) &&
              is(p_[10], type, {D, C}) && (!p_[11] || is(p_[11], type, {D})) && is(p_[8], at::kFloat, {heads_});
    for (int i = 3; i < 8; ++i) ok = ok && is(p_[i], at::kFloat, {heads_});
    ok = ok && is(conv, type, {M, C, d_conv_ - 1}) && is(state, at::kFloat, {M, heads_, P_, 2 * N_}) &&
         is(b_prev, type, {M, groups_, 2 * N_}) && is(u_prev, type, {M, heads_, P_});
    const bool block = !b_.empty(), ffn = b_.size() == 6;
    // (what the row kernel of the norm takes; a dispatch mode sees a block's products, which below pass the dispatcher by)
    if (block) ok = ok && is(b_[0], type, {D}) && D % 8 == 0 && D <= 2048 && !c10::impl::TorchDispatchModeTLS::any_modes_set();
    if (ok && ffn) {
      const int64_t F = b_[4] ? b_[4]->size(1) : 0, wide = ffn_kind_ == 1 ? 2 * F : F;
      ok = is(b_[1], type, {D}) && is(b_[2], type, {wide, D}) && (!b_[3] || is(b_[3], type, {wide})) && is(b_[4], type, {D, F}) &&
           (!b_[5] || is(b_[5], type, {D})) && F % 8 == 0;
    }
    const int io = code_of(type);
    if (!block) ok = ok && x.stride(1) == 1 && x.stride(0) % 8 == 0 && sl::skinny_supported(M, D, O, io) && sl::skinny_supported(M, C, D, io);
    if (!ok) return py::none();

    Call call(x);
    const auto st = static_cast<cudaStream_t>(call.stream());
    const Tensor b_next = groups_ == heads_ ? *b_prev : at::empty_like(*b_prev);
    auto up = [](int64_t n) { return (n + 255) / 256 * 256; };
    const int64_t n_step = up(sl_mixer_decode_step_workspace_bytes(M, heads_, P_)), need = n_step + (block ? 0 : up(M * O * 2));
    const Tensor ws = workspace && workspace->numel() >= need && workspace->device() == x.device() ? *workspace : call.bytes(need);
    auto* const base = static_cast<uint8_t*>(ws.data_ptr());
    // rows of the in_proj output -> gated values and their partial sums of squares in the workspace
    auto mixer_step = [&](const void* gate, const void* value, const void* params, const void* bc, int64_t gv, int64_t ps, int64_t bs,
                          bool dependent) {
      const sl::MixerStepArgs a{gate, value, params, bc, gv, gv, ps, bs, ptr(p_[1]), ptr(p_[2]), mptr(conv), (int)d_conv_, fptr(p_[3]),
                                fptr(p_[4]), fptr(p_[5]), fptr(p_[6]), fptr(p_[7]), &cfg_, fptr(p_[8]), mfptr(state), ptr(b_prev),
                                mptr(b_next), mptr(u_prev), base, (size_t)n_step, (int)M, (int)heads_, (int)groups_, (int)P_, (int)N_,
                                io, dependent};
      check(sl::mixer_step_launch(a, st), "mixer_step");
    };
    if (!block) {   // in_proj, step, and out_proj with the row norm inside, each behind the kernel before it
      const Tensor out = call.empty({M, D}, type);
      uint8_t* const row = base + n_step;
      const sl::SkinnyArgs in{ptr(x), x.stride(0), nullptr, 0.f, nullptr, 0, ptr(p_[0]), nullptr, row, (int)M, (int)D, (int)O, io};
      check(sl::skinny_linear(in, st), "skinny_linear");
      mixer_step(row, row + C * 2, row + 2 * C * 2, row + (2 * C + 3 * heads_) * 2, O, O, O, true);
      const sl::SkinnyArgs o{base, C, ptr(p_[9]), (float)eps_[1], sl::step_partials(base, M, heads_, P_), (int)(8 * heads_), ptr(p_[10]),
                             ptr(p_[11]), mptr(out), (int)M, (int)C, (int)D, io, true};
      check(sl::skinny_linear(o, st), "skinny_linear");
      return py::make_tuple(out, b_next, ws);
    }
    // A block: five launches where token_linear takes its products, with norm, residual and activation inside; what it does not
    // take (more than 64 rows, widths that are no multiple of 8) goes to the library.  The outputs have the bits of the composed
    // path (tested): residual stream, norms and B/C phases carry a moved last bit on from block to block, up to 1.6 % after one token
    // of six blocks of width 1024.  A token of four blocks of width 512 at batch 8: 398 us with 24 library products and 29 other
    // launches, 184 with 8 launches a block (the norms by themselves), 146 with 5: the device's chain of launches bounds it now,
    // the host needs 123 of it.
    at::AutoDispatchBelowAutograd below;
    // A product requests its rows of W while the kernel before it still runs, which is sound behind a kernel of this library only:
    // those write no parameter, and start behind everything that was queued before the token.  What the program has queued in
    // front of the token, and a library product in it, may write or still wait for a weight.  (Every block's first product an
    // ordinary launch: 160 us instead of 148 for a token of four blocks of width 512.)
    auto fresh = [&](int64_t cols) { return at::detail::empty_cuda({M, cols}, type, x.device(), c10::nullopt); };
    auto norm = [&](const Tensor& a, const Tensor& w, double eps) {
      Tensor out = fresh(D);
      check(sl_rmsnorm_fwd(ptr(a), ptr(w), (float)eps, mptr(out), M, D, io, st), "sl_rmsnorm_fwd");
      behind_own = true;
      return out;
    };
    const Tensor rows = x.contiguous();
    behind_own = behind_own && x.is_contiguous();
    auto product = [&](const Tensor& a, const Tensor& W, int64_t row, int64_t n) {   // a (rows row .. row + n of W)^T
      behind_own = false;
      return at::cuda::mm(a, at::native::as_strided_tensorimpl(W, {W.size(1), n}, {1, W.size(1)}, W.storage_offset() + row * W.size(1)));
    };
    // own kernel with what follows the product inside; false where it is left to the library
    auto fused = [&](const void* a, const Tensor& W, int64_t row, int64_t n, const OptT& bias, std::initializer_list<const Tensor*> out,
                     const Tensor* residual = nullptr, int act = -1, const Tensor* norm_w = nullptr, double eps = 0.0,
                     const float* partials = nullptr) {
      sl::TokenLinearArgs t{a, static_cast<const uint8_t*>(W.data_ptr()) + row * W.size(1) * 2, ptr(bias), {}, {},
                            residual ? ptr(*residual) : nullptr, (int)M, (int)W.size(1), (int)n, io, act == 0, act == 1};
      int i = 0;
      for (const Tensor* o : out) { t.out[i] = mptr(*o); t.width[i++] = (int)o->size(1); }
      if (norm_w) { t.norm_weight = ptr(*norm_w); t.norm_eps = (float)eps; t.partials = partials; t.n_partials = (int)(8 * heads_); }
      if (!sl::token_linear_supported(t)) return false;
      t.dependent = behind_own;
      check(sl::token_linear(t, st), "token_linear");
      return behind_own = true;
    };
    auto linear = [&](const Tensor& a, const Tensor& W, const OptT& bias) {
      behind_own = false;
      return bias ? at::linear(a, W, bias) : product(a, W, 0, W.size(0));
    };
    // residual + linear
    auto onto = [&](const Tensor& residual, const Tensor& a, const Tensor& W, const OptT& bias) {
      Tensor out = fresh(D);
      if (fused(ptr(a), W, 0, D, bias, {&out}, &residual)) return out;
      const Tensor branch = linear(a, W, bias);
      check(sl::residual_sum(ptr(residual), ptr(branch), mptr(out), M * D, io, st), "residual_sum");
      behind_own = true;
      return out;
    };
    const int64_t n_gv = 2 * C, n_par = 3 * heads_, n_bc = 4 * groups_ * N_;
    Tensor gv = fresh(n_gv), params = fresh(n_par), bc = fresh(n_bc);
    if (!fused(ptr(rows), *p_[0], 0, O, {}, {&gv, &params, &bc}, nullptr, -1, &*b_[0], eps_[0])) {
      const Tensor normed = norm(rows, *b_[0], eps_[0]);
      if (!fused(ptr(normed), *p_[0], 0, O, {}, {&gv, &params, &bc})) {
        if (!fused(ptr(normed), *p_[0], 0, n_gv, {}, {&gv})) gv = product(normed, *p_[0], 0, n_gv);
        if (!fused(ptr(normed), *p_[0], n_gv, n_par, {}, {&params})) params = product(normed, *p_[0], n_gv, n_par);
        if (!fused(ptr(normed), *p_[0], n_gv + n_par, n_bc, {}, {&bc})) bc = product(normed, *p_[0], n_gv + n_par, n_bc);
      }
    }
    mixer_step(gv.data_ptr(), column(gv, C), params.data_ptr(), bc.data_ptr(), n_gv, n_par, n_bc, false);
    behind_own = true;
    Tensor out = fresh(D);
    if (!fused(base, *p_[10], 0, D, p_[11], {&out}, &rows, -1, &*p_[9], eps_[1], sl::step_partials(base, M, heads_, P_))) {
      const Tensor hid = fresh(C);
      check(sl::mixer_step_norm(base, ptr(p_[9]), (float)eps_[1], mptr(hid), M, heads_, P_, io, st), "mixer_step");
      out = onto(rows, hid, *p_[10], p_[11]);
    }
    if (ffn) {
      const Tensor act = fresh(b_[4]->size(1));
      if (!fused(ptr(out), *b_[2], 0, b_[2]->size(0), b_[3], {&act}, nullptr, ffn_kind_, &*b_[1], eps_[2])) {
        const Tensor in = norm(out, *b_[1], eps_[2]);
        if (!fused(ptr(in), *b_[2], 0, b_[2]->size(0), b_[3], {&act}, nullptr, ffn_kind_)) {
          const Tensor wide = linear(in, *b_[2], b_[3]);
          check(sl_ffn_activation_fwd(ptr(wide), mptr(act), M, act.size(1), ffn_kind_, io, st), "sl_ffn_activation_fwd");
        }
      }
      out = onto(out, act, *b_[4], b_[5]);
    }
    return py::make_tuple(out, b_next, ws);
  }

 private:
  static TokenPlan* of(PyObject* self) {   // null while the constructor has not run
    const auto held = reinterpret_cast<py::detail::instance*>(self)->get_value_and_holder();
    return held.holder_constructed() ? static_cast<TokenPlan*>(held.value_ptr()) : nullptr;
  }

  std::vector<py::tuple> same_;
  std::vector<py::dict> empty_;
  std::vector<OptT> p_, b_;
  std::vector<double> eps_;        // pre-norm, mixer norm, FFN norm
  sl_scanprep_config cfg_;
  int64_t heads_, groups_, P_, N_, d_conv_;
  int ffn_kind_;
  bool cleared_ = false;
};

// ---- the whole mixer over a sequence ------------------------------------------------------------------------------------
// in_proj writes one buffer of rows [gate C | value C | params 3H | bc 4GN]; the kernels read their columns through the row
// stride, and the backward writes the four gradients into a buffer of the same layout, so each direction of in_proj is one
// GEMM and nothing is gathered in between.  Where 3H is not a multiple of 8 the bc columns start at the next one and rows of
// zeros stand in the weight for the columns between: the vector kernels want 16-byte rows, and a GEMM with such an extent
// runs at a fifth of its rate (247 instead of 74 us per block of width 576 with 18 heads); a copy of the weight costs 2 us.
struct MixerShape {
  int64_t batch, T, heads, groups, P, N, chunk, path;
  int64_t C() const { return heads * P; }
  int64_t rows() const { return batch * T; }
  int64_t front() const { return 2 * C() + 3 * heads; }                // columns before bc in the weight
  int64_t bc0() const { return (front() + 7) / 8 * 8; }               // ... and in the buffer
  int64_t bcn() const { return 4 * groups * N; }
  int64_t pitch() const { return (bc0() + bcn() + 7) / 8 * 8; }
  bool whole() const { return pitch() == front() + bcn(); }           // no column between or after
};
struct MixerWeights {
  Tensor in_w, dw_w, dw_b, d_skip, norm_w, out_w;
  std::array<Tensor, 5> bias;
  sl_scanprep_config cfg;
  float eps;
};
Tensor as_typed(const Tensor& t, at::ScalarType type) { return t.to(type).contiguous(); }

sl::ScanPrepArgs scanprep_args(const MixerShape& s, const MixerWeights& w, const Tensor& proj, const void* conv_in, void* conv_out) {
  const ULayout lay = u_layout(true, s.heads, s.T, s.P);
  return sl::ScanPrepArgs{column(proj, s.C()), s.pitch(), ptr(w.dw_w), ptr(w.dw_b), conv_in, conv_out, (int)w.dw_w.size(1),
                          column(proj, 2 * s.C()), s.pitch(), column(proj, s.bc0()), s.pitch(), fptr(w.bias[0]), fptr(w.bias[1]),
                          fptr(w.bias[2]), fptr(w.bias[3]), fptr(w.bias[4]), &w.cfg, lay.b, lay.h, lay.t, (int)s.batch,
                          (int)s.heads, (int)s.groups, (int)s.T, (int)s.P, (int)s.N, code_of(proj.scalar_type())};
}

struct MixerRun {
  Tensor in_w, proj, U, M, K, B, C, Y, normed, out;
  OptT states, final_state, conv, B_last, U_last;   // the last two, and the state, in x's type
};
MixerRun mixer_run(const MixerShape& s, const MixerWeights& w, const Tensor& x, const OptT& conv_in, const OptT& z0, const OptT& Bp,
                   const OptT& Up, bool save_states, bool want_state, const OptT& residual = {}) {
  Call call(x, w.in_w, w.dw_w, w.dw_b, w.d_skip, w.norm_w, w.out_w, conv_in, z0, Bp, Up);
  for (const auto& t : w.bias) call.need(t);
  const auto type = x.scalar_type();
  const auto st = static_cast<cudaStream_t>(call.stream());
  MixerRun r;
  r.in_w = w.in_w;
  if (!s.whole()) {
    const int64_t tail = s.pitch() - s.bc0() - s.bcn();
    const Tensor zero = call.zeros({8, w.in_w.size(1)}, type);
    r.in_w = at::cat({w.in_w.narrow(0, 0, s.front()), zero.narrow(0, 0, s.bc0() - s.front()), w.in_w.narrow(0, s.front(), s.bcn()),
                      zero.narrow(0, 0, tail)});
  }
  r.proj = at::mm(x, r.in_w.t());
  r.U = call.empty({s.batch, s.heads, s.T, s.P}, type);
  r.M = call.empty({s.batch, s.heads, s.T, 2}, at::kFloat);
  r.K = call.empty({s.batch, s.heads, s.T, 2, 2}, at::kFloat);
  r.B = call.empty({s.batch, s.groups, s.T, 2 * s.N}, type);
  r.C = at::empty_like(r.B);
  if (want_state) r.conv = call.empty({s.batch, s.C(), w.dw_w.size(1) - 1}, type);
  check(sl::scanprep_fwd(scanprep_args(s, w, r.proj, ptr(conv_in), mptr(r.conv)),
                         sl::ScanPrepOut{mptr(r.U), mfptr(r.M), mfptr(r.K), mptr(r.B), mptr(r.C)}, st),
        "sl_scanprep_conv_fwd");
  const auto last = want_state && !save_states ? scan_fwd_last(r.U, r.M, r.K, r.B, r.C, z0, Bp, Up, s.chunk, s.path) : c10::nullopt;
  if (last) {
    std::tie(r.Y, r.final_state, r.B_last, r.U_last) = *last;
  } else {
    std::tie(r.Y, r.final_state, r.states) =
        scan_fwd(r.U, r.M, r.K, r.B, r.C, z0, Bp, Up, s.chunk, code_of(type), want_state, s.path, save_states);
    if (want_state && !save_states) {
      r.final_state = r.final_state->to(type);
      r.B_last = r.B.select(2, s.T - 1).contiguous();
      r.U_last = r.U.select(2, s.T - 1).contiguous();
    }
  }
  r.normed = call.empty({s.rows(), s.C()}, type);
  check(sl_mixer_tail_fwd(ptr(r.Y), ptr(r.proj), s.pitch(), ptr(r.U), fptr(w.d_skip), ptr(w.norm_w), w.eps, mptr(r.normed), s.batch,
                          s.heads, s.T, s.P, code_of(type), st),
        "sl_mixer_tail_fwd");
  r.out = residual ? at::addmm(*residual, r.normed, w.out_w.t()) : at::mm(r.normed, w.out_w.t());
  return r;
}

MixerWeights mixer_weights(at::ScalarType type, const Tensor& in_w, const Tensor& dw_w, const Tensor& dw_b,
                           const std::array<Tensor, 5>& bias, const Config& cfg, const Tensor& d_skip, const Tensor& norm_w,
                           double eps, const Tensor& out_w) {
  MixerWeights w{in_w, as_typed(dw_w, type), as_typed(dw_b, type), as_typed(d_skip, at::kFloat), as_typed(norm_w, type), out_w,
                 {}, config_of(cfg), (float)eps};
  for (size_t i = 0; i < 5; ++i) w.bias[i] = as_typed(bias[i], at::kFloat);
  return w;
}

using Variables = torch::autograd::variable_list;
struct MixerFn : torch::autograd::Function<MixerFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& in_w, const Tensor& dw_w,
                        const Tensor& dw_b, const Tensor& dt_bias, const Tensor& alpha_bias, const Tensor& theta_mod_bias,
                        const Tensor& theta_bias, const Tensor& d_skip, const Tensor& norm_w, const Tensor& out_w,
                        const Tensor& theta_sign, std::vector<double> reals, std::vector<int64_t> dims, const OptT& pre_w) {
    const MixerShape s = shape_of(dims);
    const bool block = pre_w.has_value();   // x + mixer(norm(x)) instead of mixer(x)
    const Tensor stream = x.reshape({s.rows(), x.size(-1)}).contiguous();
    const Tensor flat = block ? rmsnorm_fwd(stream, *pre_w, (float)reals[11]) : stream;
    const MixerWeights w = weights_of(flat.scalar_type(), in_w, dw_w, dw_b, {dt_bias, alpha_bias, theta_mod_bias, theta_bias, theta_sign},
                                      reals, d_skip, norm_w, out_w);
    const MixerRun r = mixer_run(s, w, flat, {}, {}, {}, {}, true, false, block ? OptT(stream) : OptT());
    ctx->save_for_backward({flat, s.whole() ? in_w : r.in_w, w.dw_w, w.dw_b, w.bias[0], w.bias[1], w.bias[2], w.bias[3], w.d_skip, w.norm_w, out_w,
                            w.bias[4], r.proj, r.U, r.M, r.K, r.B, r.C, r.Y, r.normed, r.states ? *r.states : Tensor(),
                            r.states ? *r.final_state : Tensor(), block ? stream : Tensor(), block ? *pre_w : Tensor()});
    for (const Tensor& t : {dw_w, dw_b, dt_bias, alpha_bias, theta_mod_bias, theta_bias, d_skip, norm_w})
      dims.push_back((int64_t)t.scalar_type());
    auto shape = x.sizes().vec();
    ctx->saved_data["reals"] = reals;
    ctx->saved_data["dims"] = dims;
    ctx->saved_data["x"] = shape;
    shape.back() = out_w.size(0);
    return r.out.view(shape);
  }

  static Variables backward(torch::autograd::AutogradContext* ctx, Variables grads) {
    const auto v = ctx->get_saved_variables();
    const auto reals = ctx->saved_data["reals"].toDoubleVector();
    const auto dims = ctx->saved_data["dims"].toIntVector();
    const MixerShape s = shape_of(dims);
    const Tensor &x = v[0], &in_w = v[1], &out_w = v[10], &proj = v[12], &U = v[13], &Y = v[18], &normed = v[19];
    const MixerWeights w = weights_of(x.scalar_type(), in_w, v[2], v[3], {v[4], v[5], v[6], v[7], v[11]}, reals, v[8], v[9], out_w);
    OptT states, final_state;
    if (v[20].defined()) { states = v[20]; final_state = v[21]; }
    Call call(x, grads[0]);
    const auto type = x.scalar_type();
    const auto st = static_cast<cudaStream_t>(call.stream());
    Variables g(15);
    const Tensor dout = grads[0].reshape({s.rows(), grads[0].size(-1)});
    if (ctx->needs_input_grad(10)) g[10] = at::mm(dout.t(), normed);
    Tensor dn = at::mm(dout, out_w);
    // float32 accumulators of the small parameters: slices of one zeroed buffer, 16-byte aligned in every type
    const int64_t W = w.dw_w.size(1), C = s.C(), H = s.heads;
    const std::array<int64_t, 8> len{C * W, C, C, H, H, H, H, H};
    std::array<int64_t, 9> at_{};
    for (int i = 0; i < 8; ++i) at_[i + 1] = at_[i] + (len[i] + 7) / 8 * 8;
    const Tensor acc = call.zeros({at_[8]}, at::kFloat);
    auto slice = [&](int i) { return acc.narrow(0, at_[i], len[i]); };
    float* const a = mfptr(acc);
    Tensor d_proj = at::empty_like(proj), dY = at::empty_like(Y);
    check(sl::mixer_tail_bwd(ptr(Y), ptr(proj), s.pitch(), ptr(U), fptr(w.d_skip), ptr(w.norm_w), w.eps, ptr(dn), mptr(dY),
                             mptr(d_proj), s.pitch(), nullptr, a + at_[3], a + at_[2], s.batch, H, s.T, s.P, code_of(type), st),
          "sl_mixer_tail_bwd");
    dn.reset();
    {
      const auto [dU, dM, dK, dB, dC, dz, dbp, dup] =
          scan_bwd(U, v[14], v[15], v[16], v[17], {}, {}, {}, states, final_state, dY, {}, s.chunk, s.path);
      sl::ScanPrepGrads sg{ptr(dU), fptr(dM), fptr(dK), ptr(dB), ptr(dC), column(d_proj, C), s.pitch(), a + at_[0], a + at_[1],
                           nullptr, column(d_proj, 2 * C), s.pitch(), column(d_proj, s.bc0()), s.pitch(), a + at_[4], a + at_[5],
                           a + at_[6], a + at_[7]};
      sg.dY = ptr(dY);   // the skip connection's share of dU is added where dU is read
      sg.skip = fptr(w.d_skip);
      check(sl::scanprep_bwd(scanprep_args(s, w, proj, nullptr, nullptr), sg, st), "sl_scanprep_conv_bwd");
    }
    auto type_at = [&](int i) { return static_cast<at::ScalarType>(dims[8 + i]); };   // dw_w dw_b dt alpha theta_mod theta d_skip norm
    const auto t0 = type_at(0);
    if (t0 == type_at(1) && t0 == type_at(7)) {   // one conversion for the three
      const Tensor low = acc.narrow(0, 0, at_[3]).to(t0);
      g[2] = low.narrow(0, at_[0], len[0]).view({C, W});
      g[3] = low.narrow(0, at_[1], len[1]);
      g[9] = low.narrow(0, at_[2], len[2]);
    } else {
      g[2] = slice(0).view({C, W}).to(t0);
      g[3] = slice(1).to(type_at(1));
      g[9] = slice(2).to(type_at(7));
    }
    g[8] = slice(3).to(type_at(6));
    for (int i = 0; i < 4; ++i) g[4 + i] = slice(4 + i).to(type_at(2 + i));
    if (!s.whole()) {   // the columns that no kernel wrote
      const int64_t e = d_proj.element_size(), end = s.bc0() + s.bcn();
      for (const auto& [from, to] : {std::pair<int64_t, int64_t>{s.front(), s.bc0()}, {end, s.pitch()}})
        if (to > from) C10_CUDA_CHECK(cudaMemset2DAsync(column(d_proj, from), s.pitch() * e, 0, (to - from) * e, s.rows(), st));
    }
    const bool block = v[22].defined();
    if (ctx->needs_input_grad(0) || block) g[0] = at::mm(d_proj, in_w);
    if (block) std::tie(g[0], g[14]) = rmsnorm_bwd(v[22], v[23], (float)reals[11], g[0], dout.contiguous(), true);
    if (g[0].defined()) g[0] = g[0].view(ctx->saved_data["x"].toIntVector());
    if (ctx->needs_input_grad(1)) {
      g[1] = at::mm(d_proj.t(), x);
      if (!s.whole()) g[1] = at::cat({g[1].narrow(0, 0, s.front()), g[1].narrow(0, s.bc0(), s.bcn())});
    }
    return g;
  }

  static MixerShape shape_of(const std::vector<int64_t>& d) { return MixerShape{d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7]}; }
  static MixerWeights weights_of(at::ScalarType type, const Tensor& in_w, const Tensor& dw_w, const Tensor& dw_b,
                                 const std::array<Tensor, 5>& bias, const std::vector<double>& reals, const Tensor& d_skip,
                                 const Tensor& norm_w, const Tensor& out_w) {
    Config c;
    for (size_t i = 0; i < c.size(); ++i) c[i] = (float)reals[i];
    return mixer_weights(type, in_w, dw_w, dw_b, bias, c, d_skip, norm_w, reals[c.size()], out_w);
  }
};

// parameters: in_w dw_w dw_b dt_bias alpha_bias theta_mod_bias theta_bias d_skip norm_w out_w theta_sign [norm in front of the
// mixer]; reals: the ten configuration values, the norm's epsilon, and that of the norm in front; dims: heads groups P N chunk path
std::vector<int64_t> mixer_dims(const Tensor& x, const std::vector<int64_t>& dims) {
  std::vector<int64_t> d{x.size(0), x.size(1)};
  d.insert(d.end(), dims.begin(), dims.end());
  return d;
}
Tensor mixer_train(const Tensor& x, const std::vector<Tensor>& p, const std::vector<double>& reals, const std::vector<int64_t>& dims) {
  return MixerFn::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], p[9], p[10], reals, mixer_dims(x, dims),
                        p.size() > 11 ? OptT(p[11]) : OptT());
}
// without gradients: out, and on request the streaming state (conv, scan state, last B, last U)
std::tuple<Tensor, OptT, OptT, OptT, OptT> mixer_infer(const Tensor& x, const std::vector<Tensor>& p, const std::vector<double>& reals,
                                                       const std::vector<int64_t>& dims_in, const OptT& conv, const OptT& z0,
                                                       const OptT& Bp, const OptT& Up, bool want_state) {
  const auto dims = mixer_dims(x, dims_in);
  const MixerShape s = MixerFn::shape_of(dims);
  const auto type = x.scalar_type();
  const MixerWeights w = MixerFn::weights_of(type, p[0], p[1], p[2], {p[3], p[4], p[5], p[6], p[10]}, reals, p[7], p[8], p[9]);
  auto cast = [](const OptT& t, at::ScalarType ty) { return t ? OptT(as_typed(*t, ty)) : OptT(); };
  MixerRun r = mixer_run(s, w, x.reshape({s.rows(), x.size(-1)}), cast(conv, type), cast(z0, at::kFloat), cast(Bp, type),
                         cast(Up, type), false, want_state);
  Tensor out = r.out.view({s.batch, s.T, r.out.size(1)});
  if (!want_state) return {out, {}, {}, {}, {}};
  return {out, r.conv, r.final_state, r.B_last, r.U_last};
}

// ---- FFN branch of a block in training: x + W2 act(W1 norm(x) + b1) + b2 ----------------------------------------------------
// One node; the residual gradient is added where the norm's is written, and the bias gradients are column sums.
struct FFNFn : torch::autograd::Function<FFNFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& norm_w, const Tensor& w1, const Tensor& w2,
                        double eps, int64_t kind, const OptT& b1, const OptT& b2) {
    const Tensor rows = x.reshape({-1, x.size(-1)}).contiguous();
    const Tensor normed = rmsnorm_fwd(rows, norm_w, (float)eps), projected = at::linear(normed, w1, b1);
    const Tensor hidden = ffn_act_fwd(projected, (int)kind);
    const Tensor out = b2 ? rows + at::linear(hidden, w2, b2) : at::addmm(rows, hidden, w2.t());
    ctx->save_for_backward({rows, norm_w, w1, w2, normed, projected, hidden});
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["kind"] = kind;
    ctx->saved_data["b1"] = b1.has_value();
    ctx->saved_data["b2"] = b2.has_value();
    ctx->saved_data["x"] = x.sizes().vec();
    return out.view(x.sizes());
  }
  static Variables backward(torch::autograd::AutogradContext* ctx, Variables grads) {
    const auto v = ctx->get_saved_variables();
    const Tensor &rows = v[0], &norm_w = v[1], &w1 = v[2], &w2 = v[3], &normed = v[4], &projected = v[5], &hidden = v[6];
    const bool b1 = ctx->saved_data["b1"].toBool(), b2 = ctx->saved_data["b2"].toBool();
    const int64_t D = rows.size(1), W = projected.size(1), n = rows.size(0);
    const int kind = (int)ctx->saved_data["kind"].toInt(), io = code_of(rows.scalar_type());
    Variables g(8);
    const Tensor dout = grads[0].reshape({n, D}).contiguous();
    Call call(rows, dout);
    const auto st = static_cast<cudaStream_t>(call.stream());
    // float64 sums over the rows: norm weight, both biases
    const Tensor sums = call.zeros({2 * D + W}, at::kDouble);
    double* const acc = sums.data_ptr<double>();
    const bool fused_b2 = b2 && sl::rmsnorm_bwd_sums_extra(D);
    g[3] = at::mm(dout.t(), hidden);
    const Tensor d_hid = at::mm(dout, w2);
    Tensor d_proj;
    if (b1) {
      d_proj = at::empty_like(projected);
      check(sl::ffn_act_bwd_sum(ptr(projected), ptr(d_hid), mptr(d_proj), acc + 2 * D, n, hidden.size(1), kind, io, st),
            "sl_ffn_activation_bwd");
    } else {
      d_proj = ffn_act_bwd(projected, d_hid, kind);
    }
    g[2] = at::mm(d_proj.t(), normed);
    const Tensor dn = at::mm(d_proj, w1);
    g[0] = at::empty_like(rows);
    check(sl::rmsnorm_bwd(ptr(rows), ptr(norm_w), (float)ctx->saved_data["eps"].toDouble(), ptr(dn), ptr(dout), mptr(g[0]), nullptr, acc,
                          fused_b2 ? acc + D : nullptr, n, D, io, st),
          "sl_rmsnorm_bwd");
    g[0] = g[0].view(ctx->saved_data["x"].toIntVector());
    const Tensor low = sums.to(rows.scalar_type());
    g[1] = low.narrow(0, 0, D);
    if (b1) g[6] = low.narrow(0, 2 * D, W);
    if (b2) g[7] = fused_b2 ? low.narrow(0, D, D) : column_sum(dout);
    return g;
  }
};
Tensor ffn_train(const Tensor& x, const Tensor& norm_w, const Tensor& w1, const OptT& b1, const Tensor& w2, const OptT& b2, double eps,
                 int64_t kind) {
  return FFNFn::apply(x, norm_w, w1, w2, eps, kind, b1, b2);
}

// ---- language-model training step --------------------------------------------------------------------------------------
// loss, scale of the gradient and the log-sum-exps of the rows of logits (rows, V)
std::tuple<Tensor, Tensor, Tensor> ce_fwd(const Tensor& logits, const Tensor& target, bool mean) {
  Call call(logits, target);
  const int64_t rows = logits.size(0), V = logits.size(1);
  const Tensor loss = call.empty({rows}, at::kFloat), lse = call.empty({rows}, at::kFloat);
  const Tensor total = call.empty({}, at::kFloat), scale = call.empty({}, at::kFloat);
  check(sl::cross_entropy_fwd(ptr(logits), target.const_data_ptr<int64_t>(), mfptr(loss), mfptr(lse), rows, V,
                              code_of(logits.scalar_type()), static_cast<cudaStream_t>(call.stream())),
        "cross_entropy_fwd");
  check(sl::cross_entropy_finish(fptr(loss), target.const_data_ptr<int64_t>(), rows, mean, mfptr(total), mfptr(scale),
                                 static_cast<cudaStream_t>(call.stream())),
        "cross_entropy_fwd");
  return {total, scale, lse};
}
Tensor ce_bwd(const Tensor& logits, const Tensor& target, const Tensor& lse, const Tensor& g, const Tensor& scale) {
  Call call(logits, target, lse, g, scale);
  const int64_t rows = logits.size(0), V = logits.size(1);
  Tensor d = at::empty_like(logits);
  check(sl::cross_entropy_bwd(ptr(logits), target.const_data_ptr<int64_t>(), fptr(lse), fptr(g), fptr(scale), mptr(d), rows, V,
                              code_of(logits.scalar_type()), static_cast<cudaStream_t>(call.stream())),
        "cross_entropy_bwd");
  return d;
}
Tensor embed_bwd(const Tensor& ids, const Tensor& d_out, int64_t V) {
  Call call(ids, d_out);
  const int64_t n = ids.numel(), C = d_out.size(-1);
  auto [sorted, order] = at::sort(ids.reshape({-1}).to(at::kInt), c10::optional<bool>(true), 0, false);
  const Tensor rows = d_out.contiguous();
  Tensor dE = call.empty({V, C}, d_out.scalar_type());
  check(sl::embedding_bwd(sorted.const_data_ptr<int>(), order.const_data_ptr<int64_t>(), ptr(rows), mptr(dE), n, V, C,
                          code_of(d_out.scalar_type()), static_cast<cudaStream_t>(call.stream())),
        "embedding_bwd");
  return dE;
}

// {global norm, max(1, (norm + 1e-6) / clip)} of a list of tensors of up to three types
Tensor grad_norm_scale(const std::vector<Tensor>& grads, double clip) {
  if (grads.empty()) throw pybind11::value_error("no gradients.");
  Call call(grads[0]);
  for (const auto& g : grads) call.need(g);
  const auto st = static_cast<cudaStream_t>(call.stream());
  int64_t total = 0;
  for (const auto& g : grads) total += sl::mt_chunks(g.numel());
  Tensor partial = call.empty({std::max<int64_t>(total, 1)}, at::kFloat), out = call.empty({2}, at::kFloat);
  int64_t at_chunk = 0;
  for (int io : {SL_F32, SL_BF16, SL_F16}) {
    sl::MtList1 list{};
    unsigned chunks = 0;
    auto flush = [&] {
      if (!chunks) return;
      check(sl::multi_sumsq(list, chunks, mfptr(partial) + at_chunk, io, st), "grad_norm");
      at_chunk += chunks; chunks = 0; list.n = 0;
    };
    for (const auto& g : grads) {
      if (code_of(g.scalar_type()) != io || g.numel() == 0) continue;
      list.p[list.n] = ptr(g); list.len[list.n] = g.numel(); list.first[list.n] = chunks; ++list.n;
      chunks += sl::mt_chunks(g.numel());
      if (list.n == sl::MT_MAX) flush();
    }
    flush();
  }
  check(sl::norm_finish(fptr(partial), (int)at_chunk, (float)clip, mfptr(out), st), "grad_norm");
  return out;
}

// one AdamW step over lists of parameters, gradients and moments (all dense and of one type per position)
void adamw_step(const std::vector<Tensor>& ps, const std::vector<Tensor>& gs, const std::vector<Tensor>& ms,
                const std::vector<Tensor>& vs, const Tensor& step, double lr, double beta1, double beta2, double eps,
                double weight_decay, const OptT& grad_scale) {
  Call call(step, grad_scale);
  for (const auto& p : ps) call.need(p);
  const auto st = static_cast<cudaStream_t>(call.stream());
  const sl::AdamWArgs a{(float)lr, (float)eps, (float)(1.0 - lr * weight_decay), (float)beta2, (float)(1.0 - beta1),
                        (float)(1.0 - beta2), std::log(beta1), std::log(beta2), fptr(step), fptr(grad_scale)};
  for (int io : {SL_F32, SL_BF16, SL_F16}) {
    sl::MtList4 list{};
    unsigned chunks = 0;
    auto flush = [&] {
      if (chunks) check(sl::multi_adamw(list, chunks, a, io, st), "adamw");
      chunks = 0; list.n = 0;
    };
    for (size_t i = 0; i < ps.size(); ++i) {
      if (code_of(ps[i].scalar_type()) != io || ps[i].numel() == 0) continue;
      const int n = list.n++;
      list.p[n] = mptr(ps[i]); list.g[n] = mptr(gs[i]); list.m[n] = mptr(ms[i]); list.v[n] = mptr(vs[i]);
      list.len[n] = ps[i].numel(); list.first[n] = chunks;
      chunks += sl::mt_chunks(ps[i].numel());
      if (list.n == sl::MT_MAX) flush();
    }
    flush();
  }
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("scan_fwd", &scan_fwd);
  m.def("scan_fwd_last", &scan_fwd_last);
  m.def("scan_bwd", &scan_bwd);
  m.def("scan_decode", &scan_decode);
  m.def("scanprep_fwd", &scanprep_fwd);
  m.def("scanprep_bwd", &scanprep_bwd);
  m.def("tail_fwd", &tail_fwd);
  m.def("tail_bwd", &tail_bwd);
  m.def("rmsnorm_fwd", &rmsnorm_fwd);
  m.def("rmsnorm_bwd", &rmsnorm_bwd);
  m.def("column_sum", &column_sum);
  m.def("ffn_act_fwd", &ffn_act_fwd);
  m.def("ffn_act_bwd", &ffn_act_bwd);
  m.def("ce_fwd", &ce_fwd);
  m.def("ce_bwd", &ce_bwd);
  m.def("embed_bwd", &embed_bwd);
  m.def("grad_norm_scale", &grad_norm_scale);
  m.def("adamw_step", &adamw_step);
  m.def("mixer_train", &mixer_train);
  m.def("mixer_infer", &mixer_infer);
  m.def("ffn_train", &ffn_train);
  m.def("mixer_token", &mixer_token);
  // (a copied or unpickled module makes a plan of its own)
  py::class_<TokenPlan>(m, "TokenPlan", py::custom_type_setup(&TokenPlan::collectable))
      .def(py::init<std::vector<py::tuple>, std::vector<py::dict>, std::vector<OptT>, std::vector<OptT>, std::vector<double>,
                    const Config&, std::array<int64_t, 5>, int>())
      .def("valid", &TokenPlan::valid)
      .def("step", &TokenPlan::step)
      .def("__deepcopy__", [](const TokenPlan&, py::dict) { return py::none(); })
      .def("__reduce__", [](const TokenPlan&) { return py::make_tuple(py::type::of(py::none()), py::tuple()); });
}
