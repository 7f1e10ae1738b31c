"""CUDA-graph decode engine for ``SLinOSSMixer``: one captured graph per token.

A decode token of the mixer is in_proj, the step kernel (conv update, scan preparation, state update, skip,
gate, partial sums for the row norm) and out_proj.  Up to 64 rows of a 16-bit type the projections are the
small-batch kernels, the second with the row norm inside: three launches; else they are library GEMMs with
a kernel for the norm in between.  Their launches cost more host time than the GPU needs at small batch; the engine
captures them once over static buffers and replays the graph per token.  The reference has the same idea for
its whole model (scripts/perf/_training_model.py:120-200); here it is part of the package because
the fused step exists to be replayed.
"""

from __future__ import annotations

import torch

from .layers.state import SLinOSSMixerState


class MixerDecodeEngine:
    """Holds a mixer's decode state in static buffers and advances it one token per ``step``.

    ``step(x)`` takes ``x (batch, d_model)`` and returns ``y (batch, d_model)`` (a view of the engine's
    output buffer: copy it if it must outlive the next step).  ``reset()`` zeroes the carried state.
    The mixer's parameters are read at replay time, so weight updates are seen; changing their
    shapes, dtype or device needs a new engine."""

    def __init__(self, mixer, batch_size: int, *, device=None, dtype=None, use_graph: bool = True):
        p = next(mixer.parameters())
        self.mixer = mixer
        self.device = torch.device(device) if device is not None else p.device
        self.dtype = dtype or p.dtype
        if self.device.type != "cuda":
            raise ValueError("MixerDecodeEngine needs a CUDA device: the kernels have no CPU path.")
        from . import _C
        self.batch = int(batch_size)
        self.state: SLinOSSMixerState = mixer.init_decode_state(self.batch, device=self.device, dtype=self.dtype)
        kw = dict(device=self.device, dtype=self.dtype)
        self.x = torch.zeros((self.batch, mixer.d_model), **kw)
        self.y = torch.zeros((self.batch, mixer.d_model), **kw)
        self._b_prev = self.state.scan.b_prev    # (the step hands the new one on in a tensor of its own when heads share groups)
        self._workspace = _C.mixer_decode_workspace(self.batch, mixer.n_heads, mixer.d_head, self.device)
        self._graph = None
        if use_graph:
            self._capture()

    # one token over the static buffers (everything in place: the graph sees fixed addresses)
    def _token(self):
        st = self.state
        self.mixer.decode_native(self.x, st, workspace=self._workspace, out=self.y)
        if st.scan.b_prev is not self._b_prev:
            self._b_prev.copy_(st.scan.b_prev)
            st.scan.b_prev = self._b_prev

    def _capture(self):
        side = torch.cuda.Stream(self.device)
        side.wait_stream(torch.cuda.current_stream(self.device))
        with torch.cuda.stream(side), torch.no_grad():      # warm-up outside the capture
            self._token()
        torch.cuda.current_stream(self.device).wait_stream(side)
        torch.cuda.synchronize(self.device)
        self.reset()
        self._graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(self._graph):
            self._token()
        torch.cuda.synchronize(self.device)
        self.reset()

    def reset(self):
        st = self.state
        for t in (st.conv, st.scan.state, st.scan.b_prev, st.scan.u_prev):
            t.zero_()

    @torch.no_grad()
    def step(self, x: torch.Tensor) -> torch.Tensor:
        if tuple(x.shape) != tuple(self.x.shape):
            raise ValueError(f"Expected x shape {tuple(self.x.shape)}, got {tuple(x.shape)}.")
        self.x.copy_(x)
        if self._graph is not None:
            self._graph.replay()
        else:
            self._token()
        return self.y


__all__ = ["MixerDecodeEngine"]
