"""Pre-norm residual block: ``x + mixer(norm(x))`` then ``x + ffn(norm(x))``.

Composition, parameter names and residual arithmetic (float32 add, cast back)
follow the reference block (slinoss/blocks/block.py:41-303).  On CUDA the FFN
branch runs as one rematerialising op (``ops.block.ffn_residual``) when its
conditions hold, else as plain torch.
"""

from __future__ import annotations

import torch
import torch.nn.functional as F
from torch import nn

from .. import _C
from ..layers import RMSNorm, SLinOSSMixer
from ..layers.mixer import _norm_eps, planned_step
from ..layers.mlp import SLinOSSMLP
from ..ops.block import ffn_residual, ffn_residual_supported, residual_add
from .config import SLinOSSBlockConfig
from .state import SLinOSSBlockState


def make_norm(kind, d_model, *, eps, device=None, dtype=None) -> nn.Module:
    if kind == "rmsnorm":
        return RMSNorm(d_model, eps=eps, device=device, dtype=dtype)
    return nn.LayerNorm(d_model, eps=eps, device=device, dtype=dtype)


def apply_norm(norm: nn.Module, x: torch.Tensor) -> torch.Tensor:
    w = getattr(norm, "weight", None)
    return norm(x.to(dtype=w.dtype)) if isinstance(w, torch.Tensor) else norm(x)


def _plain_rmsnorm(norm, x) -> bool:
    if type(norm) is not RMSNorm or norm._forward_hooks or norm._forward_pre_hooks:
        return False
    w = norm._parameters["weight"]
    return (w is not None and w.dtype == x.dtype and w.device == x.device and w.shape == x.shape[-1:]
            and x.dtype in (torch.bfloat16, torch.float16) and _C.rmsnorm_supported(int(x.shape[-1]), x.dtype))


def _plain_linear(layer, x) -> bool:
    w, b = layer._parameters["weight"], layer._parameters["bias"]
    return (type(layer) is nn.Linear and not layer._forward_hooks and not layer._forward_pre_hooks
            and w.dtype == x.dtype and w.device == x.device and w.is_contiguous()
            and (b is None or b.dtype == x.dtype))


@_C.opaque
def _ffn_train(x, norm, ffn):
    """``x + ffn(norm(x))`` as one autograd node."""
    w1, w2 = ffn.in_proj._parameters, ffn.out_proj._parameters
    return _C.host().ffn_train(x, norm.weight, w1["weight"], w1["bias"], w2["weight"], w2["bias"], _norm_eps(norm),
                               _C.FFN_KINDS[ffn.kind])


class SLinOSSBlock(nn.Module):
    def __init__(self, config: SLinOSSBlockConfig, *, device=None, dtype=None) -> None:
        super().__init__()
        self.config, self.d_model = config, config.d_model
        self.residual_in_fp32 = bool(config.residual_in_fp32)
        self.residual_dropout = float(config.residual_dropout)
        # What the FFN branch rebuilds in the backward pass on CUDA: "full" (keeps only the branch input,
        # the reference's schedule), "rows" (keeps the projection too: no GEMM is repeated) or "none"
        # (plain autograd, the default: fastest while the activations fit in memory).
        self.ffn_remat = "none"
        kw = {"device": device, "dtype": dtype}
        self.mixer_norm = make_norm(config.norm_kind, config.d_model, eps=config.norm_eps, **kw)
        self.mixer = SLinOSSMixer(config.d_model, **config.mixer.build_kwargs(), **kw)
        if config.ffn is None:
            self.ffn_norm, self.ffn = None, None
        else:
            self.ffn_norm = make_norm(config.norm_kind, config.d_model, eps=config.norm_eps, **kw)
            self.ffn = SLinOSSMLP.from_config(config.d_model, config.ffn, **kw)

    def init_state(self, batch_size, *, device=None, dtype=None) -> SLinOSSBlockState:
        return SLinOSSBlockState(mixer=self.mixer.init_state(batch_size, device=device, dtype=dtype))

    def init_decode_state(self, batch_size, *, device=None, dtype=None) -> SLinOSSBlockState:
        return SLinOSSBlockState(
            mixer=self.mixer.init_decode_state(batch_size, device=device, dtype=dtype))

    def _drop(self, x):
        return x if self.residual_dropout <= 0.0 else F.dropout(x, self.residual_dropout, self.training)

    def _add(self, residual, branch):
        return residual_add(residual, branch, self.residual_in_fp32)

    def _native_training_ready(self, x) -> bool:
        """The mixer branch with its norm and residual as one node: gradients wanted, one 16-bit type, no dropout, no hooks."""
        mixer = self.mixer
        return (x.is_cuda and torch.is_grad_enabled() and (self.residual_dropout <= 0.0 or not self.training)
                and type(mixer) is SLinOSSMixer and not mixer._forward_hooks and not mixer._forward_pre_hooks
                and not mixer._backward_hooks and not mixer._backward_pre_hooks and _plain_rmsnorm(self.mixer_norm, x)
                and mixer._native_forward_ready(x, None))

    def _ffn_residual(self, x):
        no_drop = self.residual_dropout <= 0.0 or not self.training
        ffn, norm = self.ffn, self.ffn_norm
        if no_drop and self.ffn_remat == "none" and x.is_cuda and torch.is_grad_enabled() and type(ffn) is SLinOSSMLP \
                and not (ffn._forward_hooks or ffn._forward_pre_hooks or ffn._backward_hooks or ffn._backward_pre_hooks) \
                and _plain_rmsnorm(norm, x) and _plain_linear(ffn.in_proj, x) and _plain_linear(ffn.out_proj, x) \
                and ffn_residual_supported(x, norm, ffn):
            return _ffn_train(x, norm, ffn)
        if no_drop and self.ffn_remat != "none" and ffn_residual_supported(x, self.ffn_norm, self.ffn):
            return ffn_residual(x, self.ffn_norm, self.ffn, residual_in_fp32=self.residual_in_fp32,
                                remat=self.ffn_remat)
        return self._add(x, self._drop(self.ffn(apply_norm(self.ffn_norm, x))))

    def forward(self, x, *, state: SLinOSSBlockState | None = None, return_state: bool = False,
                context=None, sequence_group=None):
        if x.ndim != 3 or x.shape[-1] != self.d_model:
            raise ValueError(f"Expected x shape (batch, T, {self.d_model}), got {tuple(x.shape)}.")
        if state is None and not return_state and sequence_group is None and self._native_training_ready(x):
            out = self.mixer._forward_native(x, self.mixer._native_parameters(), None, False, pre_norm=self.mixer_norm)
            return out if self.ffn is None else self._ffn_residual(out)
        extra = {} if sequence_group is None else {"sequence_group": sequence_group}
        mixed = self.mixer(apply_norm(self.mixer_norm, x),
                           state=None if state is None else state.mixer, return_state=return_state, **extra)
        nxt = None
        if return_state:
            mixed, mixer_state = mixed
            nxt = SLinOSSBlockState(mixer=mixer_state)
        out = self._add(x, self._drop(mixed))
        if self.ffn is not None:
            out = self._ffn_residual(out)
        return (out, nxt) if return_state else out

    def _make_token_plan(self):
        mixer, ffn, norm = self.mixer, self.ffn, self.mixer_norm
        kids = self._modules
        if type(norm) is not RMSNorm or norm.weight is None or norm.eps is None:
            return None
        # (None: this block's __dict__, which keeps the plan)
        same = [(kids, n, kids[n]) if n in kids else (None, n, self.__dict__[n])
                for n in ("mixer", "mixer_norm", "ffn", "ffn_norm")]
        same += [(norm._parameters, "weight", norm.weight), (norm.__dict__, "eps", norm.eps), (norm.__dict__, "forward")]
        empty = [mixer._forward_hooks, mixer._forward_pre_hooks, norm._forward_hooks, norm._forward_pre_hooks]
        branch, ffn_eps, kind = [norm.weight], 0.0, 0
        if ffn is not None:
            fnorm = self.ffn_norm
            if not (type(ffn) is SLinOSSMLP and type(fnorm) is RMSNorm and fnorm.weight is not None and fnorm.eps is not None
                    and type(ffn.in_proj) is nn.Linear and type(ffn.out_proj) is nn.Linear):
                return None
            same += [(ffn._modules, n, ffn._modules[n]) for n in ("in_proj", "out_proj")]
            same += [(ffn.__dict__, "kind", ffn.kind), (fnorm._parameters, "weight", fnorm.weight), (fnorm.__dict__, "eps", fnorm.eps)]
            for layer in (ffn.in_proj, ffn.out_proj):
                same += [(layer._parameters, n, layer._parameters[n]) for n in ("weight", "bias")]
            for m in (ffn, fnorm, ffn.in_proj, ffn.out_proj):
                empty += [m._forward_hooks, m._forward_pre_hooks]
                same.append((m.__dict__, "forward"))
            branch += [fnorm.weight, ffn.in_proj.weight, ffn.in_proj.bias, ffn.out_proj.weight, ffn.out_proj.bias]
            ffn_eps, kind = _norm_eps(fnorm), _C.FFN_KINDS[ffn.kind]
        return mixer._make_token_plan(branch, (same, empty), _norm_eps(norm), ffn_eps, kind)

    def _native_step(self, token, state, inplace, behind=False):
        """The whole step through the block's native plan (the composed path's products and kernels as one call), or None when
        something asks for the composed path: gradients, another norm, dropout, autocast, hooks, an injected backend, a
        partial state."""
        if torch.is_grad_enabled() or state is None or not token.is_cuda or (inplace is not None and not inplace) or \
                (self.residual_dropout > 0.0 and self.training) or type(self.mixer) is not SLinOSSMixer:
            return None
        out = planned_step(self, token, state.mixer, self._make_token_plan, behind)
        return None if out is None else (out, SLinOSSBlockState(mixer=state.mixer))

    def step(self, x, state: SLinOSSBlockState | None = None, *, inplace=None, context=None):
        return self._advance(x, state, inplace)[:2]

    def _advance(self, x, state, inplace, behind=False):
        """``step``, and whether its last kernel is the plan's own (``behind`` of a block right after this one)."""
        token = x
        if token.ndim == 3:
            if token.shape[1] != 1:
                raise ValueError(f"Expected time dim 1 for block.step, got {tuple(token.shape)}.")
            token = token[:, 0, :]
        if token.ndim != 2 or token.shape[-1] != self.d_model:
            raise ValueError(f"Expected x shape (batch, {self.d_model}) or "
                             f"(batch, 1, {self.d_model}), got {tuple(x.shape)}.")
        done = self._native_step(token, state, inplace, behind)
        if done is not None:
            return done[0] if x.ndim == 2 else done[0].unsqueeze(1), done[1], True
        normed, carried, mixer = apply_norm(self.mixer_norm, token), None if state is None else state.mixer, self.mixer
        if type(mixer) is SLinOSSMixer and "step" not in mixer.__dict__:
            mixed, mixer_state = mixer._step(normed, carried, inplace, True)
        else:
            mixed, mixer_state = mixer.step(normed, carried, inplace=inplace)
        out = self._add(token, self._drop(mixed.to(dtype=token.dtype)))
        if self.ffn is not None:
            out = self._ffn_residual(out)
        if x.ndim == 3:
            out = out.unsqueeze(1)
        return out, SLinOSSBlockState(mixer=mixer_state), False


PLAIN_STEP = SLinOSSBlock.step    # (a replaced method is called)

__all__ = ["SLinOSSBlock", "apply_norm", "make_norm"]
