"""ctypes binding of ``libslinoss_b200.so`` (the C-ABI CUDA library).

Two layers live here:

* ``lib()`` loads the shared library built in-tree by ``slinoss_b200.build`` and
  declares the prototypes of every ``sl_*`` symbol of ``include/slinoss_b200.h``.
  There is no fallback: if the library is missing, ``lib()`` raises.
* tensor-level launchers (``scan_fwd``, ``scan_bwd``, ``scan_decode``,
  ``scanprep_conv_fwd`` ...): names and defaults for the functions of the native host
  module (``csrc/host.cpp``), which allocate outputs and scratch with torch, launch on
  torch's *current stream* and turn non-zero status codes into exceptions.  The ops in
  ``slinoss_b200.ops`` only talk to these launchers.
"""

from __future__ import annotations

import ctypes
import functools
from ctypes import c_float, c_int, c_int64, c_size_t, c_void_p
from pathlib import Path

import torch

_LIB_PATH = Path(__file__).resolve().parent / "_lib" / "libslinoss_b200.so"
_lib = None

SL_F32, SL_BF16, SL_F16 = 0, 1, 2
PATH_AUTO, PATH_SIMT, PATH_TC = 0, 1, 2
WS_SCAN_FWD, WS_SCAN_BWD, WS_SCAN_STATES = 0, 1, 4

_DTYPE_CODE = {torch.float32: SL_F32, torch.bfloat16: SL_BF16, torch.float16: SL_F16}
_PATHS = {"auto": PATH_AUTO, "simt": PATH_SIMT, "tc": PATH_TC}


class ScanPrepConfig(ctypes.Structure):
    _fields_ = [(n, c_float) for n in (
        "dt_min", "dt_max", "alpha_min", "alpha_max", "theta_init_min", "theta_init_max",
        "theta_mod_scale", "r_min", "r_max", "eps")]


_P = c_void_p
_PROTOTYPES = {
    "sl_version": (c_int, []),
    "sl_kernel_launches": (ctypes.c_ulonglong, []),
    "sl_device_status": (c_int, []),
    "sl_device_status_reset": (c_int, []),
    "sl_status_string": (ctypes.c_char_p, [c_int]),
    "sl_last_cuda_error": (ctypes.c_char_p, []),
    "sl_workspace_bytes": (c_size_t, [c_int] * 10),
    "sl_v2x2ssd_fwd": (c_int, [_P] * 11 + [c_int] * 10 + [_P, c_size_t, _P]),
    "sl_v2x2ssd_bwd": (c_int, [_P] * 20 + [c_int] * 10 + [_P, c_size_t, _P]),
    "sl_static_scratch_bytes": (c_size_t, []),
    "sl_v2x2ssd_bwd_static": (c_int, [_P] * 18 + [c_int] * 8 + [_P]),
    "sl_v2x2ssd_decode": (c_int, [_P] * 10 + [c_int] * 7 + [_P]),
    "sl_scanprep_conv_fwd": (c_int, [_P, c_int64, _P, _P, _P, _P, c_int, _P, _P, _P, _P, _P, _P, _P,
                                     ctypes.POINTER(ScanPrepConfig), _P, c_int64, c_int64, c_int64,
                                     _P, _P, _P, _P] + [c_int] * 7 + [_P]),
    "sl_scanprep_conv_bwd": (c_int, [_P, c_int64, _P, _P, _P, c_int, _P, _P, _P, _P, _P, _P, _P,
                                     ctypes.POINTER(ScanPrepConfig), _P, c_int64, c_int64, c_int64,
                                     _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _P]
                             + [c_int] * 7 + [_P]),
    "sl_mixer_decode_step_workspace_bytes": (c_size_t, [c_int] * 3),
    "sl_mixer_decode_step": (c_int, [_P, c_int64, _P, c_int64, _P, _P, _P, _P, _P, c_int, _P, _P, _P, _P, _P,
                                     ctypes.POINTER(ScanPrepConfig), _P, _P, c_float, _P, _P, _P, _P, _P, _P,
                                     c_size_t] + [c_int] * 6 + [_P]),
    "sl_rmsnorm_fwd": (c_int, [_P, _P, c_float, _P, ctypes.c_longlong, c_int, c_int, _P]),
    "sl_rmsnorm_bwd": (c_int, [_P, _P, c_float, _P, _P, _P, ctypes.c_longlong, c_int, c_int, _P]),
    "sl_ffn_activation_fwd": (c_int, [_P, _P, ctypes.c_longlong, c_int, c_int, c_int, _P]),
    "sl_ffn_activation_bwd": (c_int, [_P, _P, _P, ctypes.c_longlong, c_int, c_int, c_int, _P]),
    "sl_mixer_tail_fwd": (c_int, [_P, _P, c_int64, _P, _P, _P, c_float, _P] + [c_int] * 5 + [_P]),
    "sl_mixer_tail_bwd": (c_int, [_P, _P, c_int64, _P, _P, _P, c_float, _P, _P, _P, _P, _P, _P]
                          + [c_int] * 5 + [_P]),
}
EXPORTED_SYMBOLS = tuple(_PROTOTYPES)


def lib_path() -> Path:
    return _LIB_PATH


def lib():
    """The loaded C-ABI library.  Raises if it has not been built."""
    global _lib
    if _lib is None:
        if not _LIB_PATH.exists():
            raise RuntimeError(
                f"slinoss_b200: CUDA library {_LIB_PATH} is missing. Build it with "
                "`python -m slinoss_b200.build` (needs nvcc); there is no fallback path.")
        handle = ctypes.CDLL(str(_LIB_PATH))
        for name, (restype, argtypes) in _PROTOTYPES.items():
            fn = getattr(handle, name)
            fn.restype = restype
            fn.argtypes = argtypes
        _lib = handle
    return _lib


_HOST_PATH = _LIB_PATH.parent / "_host.so"
_host_module = None


def host():
    """The native host module (the launchers for torch tensors).  Raises if it has not been built."""
    global _host_module
    if _host_module is None:
        lib()
        if not _HOST_PATH.exists():
            raise RuntimeError(
                f"slinoss_b200: host module {_HOST_PATH} is missing. Build it with "
                "`python -m slinoss_b200.build`; there is no fallback path.")
        import importlib.util
        spec = importlib.util.spec_from_file_location("_host", _HOST_PATH)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        _host_module = module
    return _host_module


def opaque(fn):
    """Keep ``fn`` out of ``torch.compile`` graphs.  ``torch.compiler.disable`` alone costs 3 us on every eager call;
    here the eager call goes straight through and only a trace meets the disabled function."""
    disabled = torch.compiler.disable(fn)

    @functools.wraps(fn)
    def call(*args, **kwargs):
        return disabled(*args, **kwargs) if torch.compiler.is_compiling() else fn(*args, **kwargs)
    return call


def grad_needed(*tensors) -> bool:
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def as_f32(t: torch.Tensor) -> torch.Tensor:
    """``t`` itself when it is dense float32 already, else a float32 copy."""
    return t if t.dtype is torch.float32 and t.is_contiguous() else t.detach().to(torch.float32).contiguous()


def as_type(t, dtype):
    """``t`` itself when it is dense and of ``dtype`` already (or None), else a copy."""
    return t if t is None or (t.dtype is dtype and t.is_contiguous()) else t.detach().to(dtype).contiguous()


def kernel_launches() -> int:
    """Kernels launched by the library in this process so far."""
    return int(lib().sl_kernel_launches())


def device_status() -> int:
    """0, or the status code SL_ERR_DEVICE_TIMEOUT (7) if a kernel gave up a bounded wait since
    the last reset; synchronises."""
    return int(lib().sl_device_status())


def device_status_reset() -> int:
    """Site code of the first expired wait (0 = none); clears the record; synchronises."""
    return int(lib().sl_device_status_reset())


def check(status: int, what: str) -> None:
    if status != 0:
        text = lib().sl_status_string(status).decode()
        if status == 6:   # SL_ERR_LAUNCH_FAILED: add the CUDA runtime's own words
            text += f" ({lib().sl_last_cuda_error().decode()})"
        raise RuntimeError(f"slinoss_b200.{what} failed with status {status}: {text}")


def dtype_code(dtype: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dtype]
    except KeyError:
        raise ValueError(f"unsupported dtype {dtype}; expected float32, bfloat16 or float16") from None


def require_cuda(*tensors) -> torch.device:
    """All tensors must live on one CUDA device (the kernels have no CPU path)."""
    dev = None
    for t in tensors:
        if t is None:
            continue
        if t.device.type != "cuda":
            raise ValueError("slinoss_b200 kernels require CUDA tensors.")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise ValueError("All tensors must be on the same device.")
    return dev


def _ptr(t):
    return None if t is None else t.data_ptr()


def _stream(dev) -> int:
    return torch.cuda.current_stream(dev).cuda_stream


def workspace_bytes(kind, batch, heads, groups, T, P, N, chunk, io_dtype, path="auto") -> int:
    return int(lib().sl_workspace_bytes(kind, batch, heads, groups, T, P, N, chunk,
                                        dtype_code(io_dtype), _PATHS[path]))


# ---------------------------------------------------------------------------------
# scan
# ---------------------------------------------------------------------------------
def scan_fwd(U, M, K, B, C, z0, B_prev, U_prev, *, chunk_size, y_dtype, want_final, path="auto",
             save_states=False):
    """Launch ``sl_v2x2ssd_fwd``.  ``U,B,C,B_prev,U_prev`` share one dtype; ``M,K,z0``
    are float32.  Returns ``(Y, final_state or None)``; with ``save_states`` a third item:
    the chunk-state buffer for ``scan_bwd`` (None when the chosen path keeps none)."""
    out = host().scan_fwd(U, M, K, B, C, z0, B_prev, U_prev, chunk_size, dtype_code(y_dtype), want_final,
                          _PATHS[path], save_states)
    return out if save_states else out[:2]


def scan_fwd_last(U, M, K, B, C, z0, B_prev, U_prev, *, chunk_size, path="auto"):
    """The forward scan of 16-bit operands with what a caller carries on from, all in their type: ``(Y, final_state, B_last,
    U_last)``.  None where the tensor-core path does not run."""
    if U.dtype is torch.float32 or not U.is_cuda:
        return None
    return host().scan_fwd_last(U, M, K, B, C, z0, B_prev, U_prev, chunk_size, _PATHS[path])


def scan_bwd(U, M, K, B, C, z0, B_prev, U_prev, dY, d_final, *, chunk_size, path="auto",
             saved=None):
    """Launch ``sl_v2x2ssd_bwd``.  Returns ``(dU, dM, dK, dB, dC, d_initial, dB_prev,
    dU_prev)``; the last three are None when the matching input is absent.  ``saved`` is
    ``(chunk_states, final_state)`` from ``scan_fwd(..., save_states=True)`` or None."""
    states, zfinal = saved if (saved is not None and saved[0] is not None) else (None, None)
    return host().scan_bwd(U, M, K, B, C, z0, B_prev, U_prev, states, zfinal, dY, d_final, chunk_size, _PATHS[path])


def scan_bwd_static(U, M, K, B, C, z0, B_prev, U_prev, dY, d_final, outs):
    """Launch ``sl_v2x2ssd_bwd_static``: the float32 backward with its scratch in the
    library's built-in array, for callers that may not allocate device memory.

    Nothing is allocated here either: ``outs`` is the tuple of caller-provided result
    tensors ``(dU, dM, dK, dB, dC, d_initial, dB_prev, dU_prev)`` (the last three may be
    None).  Calls share the one scratch array, so keep them on one stream."""
    dev = require_cuda(U, M, K, B, C, z0, B_prev, U_prev, dY, d_final, *outs)
    batch, heads, T, P = U.shape
    groups, N = B.shape[1], B.shape[3] // 2
    dy_code = dtype_code(dY.dtype) if dY is not None else dtype_code(U.dtype)
    with torch.cuda.device(dev):
        check(lib().sl_v2x2ssd_bwd_static(
            _ptr(U), _ptr(M), _ptr(K), _ptr(B), _ptr(C), _ptr(z0), _ptr(B_prev), _ptr(U_prev),
            _ptr(dY), _ptr(d_final), *[_ptr(o) for o in outs], batch, heads, groups, T, P, N,
            dtype_code(U.dtype), dy_code, _stream(dev)), "sl_v2x2ssd_bwd_static")
    return outs


def scan_decode(U, M, K, B, C, state, B_prev, U_prev, *, y_dtype, state_out=None):
    """Launch ``sl_v2x2ssd_decode``: one token over the carried float32 state.
    ``state_out`` defaults to a fresh tensor; pass ``state`` itself to update in place."""
    return host().scan_decode(U, M, K, B, C, state, B_prev, U_prev, dtype_code(y_dtype), state_out)


# ---------------------------------------------------------------------------------
# scan preparation (+ causal conv)
# ---------------------------------------------------------------------------------
def make_config(owner) -> ScanPrepConfig:
    return ScanPrepConfig(owner.dt_min, owner.dt_max, owner.alpha_min, owner.alpha_max,
                          owner.theta_init_min, owner.theta_init_max, owner.theta_mod_scale,
                          owner.r_min, owner.r_max, owner.eps)


CONFIG_FIELDS = tuple(n for n, _ in ScanPrepConfig._fields_)


def _config_values(cfg):
    return None if cfg is None else [getattr(cfg, n) for n in CONFIG_FIELDS]


def _row_stride(x: torch.Tensor) -> int:
    """Row stride (elements) of a (batch, T, C) tensor whose channels are dense and
    whose batch stride is T * row stride (a column slice of a dense buffer)."""
    if x.stride(2) != 1 or (x.shape[0] > 1 and x.stride(0) != x.shape[1] * x.stride(1)):
        raise ValueError(f"expected a row-strided (batch,T,C) tensor, got strides {x.stride()}")
    return int(x.stride(1)) if x.shape[1] > 1 else max(int(x.stride(1)), int(x.shape[2]))


def as_rows(x: torch.Tensor) -> torch.Tensor:
    """Return ``x`` (batch,T,C) in a layout `_row_stride` accepts, copying only if needed."""
    if x.stride(2) == 1 and (x.shape[0] == 1 or x.stride(0) == x.shape[1] * x.stride(1)) \
            and (x.shape[1] > 1 or x.stride(1) >= x.shape[2]):
        return x
    return x.contiguous()


def scanprep_conv_fwd(value, conv_weight, conv_bias, conv_state, params, bc, biases, cfg, *,
                      heads, P, u_layout="bhtp", want_state=False):
    """Launch ``sl_scanprep_conv_fwd``.

    ``value`` (batch,T,heads*P) row-strided or None; ``params`` (batch,T,3*heads) or None;
    ``bc`` (batch,T,groups,4,N) or None; ``biases`` = (dt_bias, alpha_bias, theta_mod_bias,
    theta_bias, theta_sign).  Returns ``(U, M, K, B, C, next_conv_state)`` with None for
    skipped parts.  ``u_layout`` "bhtp" gives (batch,heads,T,P), "btc" (batch,T,heads*P)."""
    return host().scanprep_fwd(value, conv_weight, conv_bias, conv_state, params, bc, biases or (),
                               _config_values(cfg), heads, P, u_layout == "bhtp", want_state)


def scanprep_conv_bwd(value, conv_weight, conv_bias, conv_state, params, bc, biases, cfg, dU, dM,
                      dK, dBo, dCo, *, heads, P, u_layout="bhtp", want_dstate=False):
    """Launch ``sl_scanprep_conv_bwd``.  Returns a dict with d_value, d_conv_weight,
    d_conv_bias, d_conv_state, d_params, d_bc, d_dt_bias, d_alpha_bias,
    d_theta_mod_bias, d_theta_bias (None for skipped parts; bias / weight gradients
    are float32 accumulators)."""
    out = host().scanprep_bwd(value, conv_weight, conv_bias, conv_state, params, bc, biases or (),
                              _config_values(cfg), dU, dM, dK, dBo, dCo, heads, P, u_layout == "bhtp", want_dstate)
    return dict(zip(("d_value", "d_conv_weight", "d_conv_bias", "d_conv_state", "d_params", "d_bc", "d_dt_bias",
                     "d_alpha_bias", "d_theta_mod_bias", "d_theta_bias"), out))


# ---------------------------------------------------------------------------------
# mixer tail (row-wise part)
# ---------------------------------------------------------------------------------
def mixer_tail_fwd(Y, gate, skip, d_skip, norm_weight, eps):
    """Launch ``sl_mixer_tail_fwd``.  Returns normed (batch,T,heads*P)."""
    return host().tail_fwd(Y, gate, skip, d_skip, norm_weight, eps)


def mixer_tail_bwd(Y, gate, skip, d_skip, norm_weight, eps, d_normed):
    """Launch ``sl_mixer_tail_bwd``.  Returns ``(dY, d_gate, d_skip_input, d_d_skip,
    d_norm_weight)``; the last two are float32 accumulators."""
    return host().tail_bwd(Y, gate, skip, d_skip, norm_weight, eps, d_normed)


# ---------------------------------------------------------------------------------
# fused decode step of the mixer
# ---------------------------------------------------------------------------------
def mixer_decode_workspace(batch, heads, P, dev) -> torch.Tensor:
    """Scratch for ``mixer_decode_step`` (allocate once, reuse every token; its content does not matter)."""
    n = lib().sl_mixer_decode_step_workspace_bytes(batch, heads, P)
    return torch.empty(n, dtype=torch.uint8, device=dev)


def mixer_decode_step(gate, value, params, bc, conv_weight, conv_bias, conv_state, biases, cfg, d_skip,
                      norm_weight, eps, state, b_prev_in, b_prev_out, u_prev, workspace, *, heads, P,
                      normed=None):
    """Call ``sl_mixer_decode_step`` (the step and its row norm: two launches).  ``gate`` and ``value`` are (batch, heads*P) views with a row
    stride; ``conv_state``, ``state`` and ``u_prev`` are updated in place; ``b_prev_out`` receives this
    token's b.  Returns ``normed`` (batch, heads*P)."""
    dev = require_cuda(gate, value, params, bc, conv_weight, conv_bias, conv_state, d_skip, norm_weight, state,
                       b_prev_in, b_prev_out, u_prev, workspace)
    batch = int(gate.shape[0])
    groups, N = int(bc.shape[-3]), int(bc.shape[-1])
    if gate.stride(-1) != 1 or value.stride(-1) != 1:
        raise ValueError("gate and value must have dense channels (row-strided views are fine).")
    if normed is None:
        normed = torch.empty((batch, heads * P), dtype=gate.dtype, device=dev)
    d_conv = 1 if conv_weight is None else int(conv_weight.shape[1])
    with torch.cuda.device(dev):
        check(lib().sl_mixer_decode_step(
            _ptr(gate), int(gate.stride(0)), _ptr(value), int(value.stride(0)), _ptr(params), _ptr(bc),
            _ptr(conv_weight), _ptr(conv_bias), _ptr(conv_state), d_conv, *[_ptr(b) for b in biases],
            ctypes.byref(cfg), _ptr(d_skip), _ptr(norm_weight), float(eps), _ptr(state), _ptr(b_prev_in),
            _ptr(b_prev_out), _ptr(u_prev), _ptr(normed), _ptr(workspace), workspace.numel(), batch, heads,
            groups, P, N, dtype_code(gate.dtype), _stream(dev)), "sl_mixer_decode_step")
    return normed


# ---------------------------------------------------------------------------------
# FFN branch: row-wise kernels
# ---------------------------------------------------------------------------------
FFN_KINDS = {"gelu": 0, "swiglu": 1}


def rmsnorm_supported(C: int, dtype: torch.dtype) -> bool:
    v = 4 if dtype == torch.float32 else 8
    return dtype in _DTYPE_CODE and C % v == 0 and C // v <= 256


def rmsnorm_fwd(x, weight, eps):
    """``x (..., C)`` dense -> same shape; launches ``sl_rmsnorm_fwd``."""
    return host().rmsnorm_fwd(x, weight, eps)


def rmsnorm_bwd(x, weight, eps, d_out, *, extra=None, as_rows_type=False):
    """Returns ``(d_x (+ extra), d_weight float32)``, the latter in x's type with ``as_rows_type``."""
    return host().rmsnorm_bwd(x, weight, eps, d_out, extra, as_rows_type)


def column_sum(x):
    """Sum over all but the last axis in float32, rounded once to x's type."""
    return host().column_sum(x)


def ffn_activation_fwd(projected, kind: str):
    """``projected (..., W)`` dense, W = hidden (gelu) or 2*hidden (swiglu) -> ``hidden (..., hidden)``."""
    return host().ffn_act_fwd(projected, FFN_KINDS[kind])


def ffn_activation_bwd(projected, d_hidden, kind: str):
    return host().ffn_act_bwd(projected, d_hidden, FFN_KINDS[kind])
