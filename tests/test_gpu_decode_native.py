"""The native decode step of a block (small-batch linear kernels, pipelined state update) against the composed path:
library GEMMs, row kernels, and conv, scan preparation, decode and tail as launches of their own."""

import pytest
import torch

import slinoss_b200 as sb
from slinoss_b200 import _C
from tests.util import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _block(d_model, state, groups, kind, bias, dtype):
    torch.manual_seed(1)
    cfg = sb.SLinOSSBlockConfig(d_model=d_model,
                                mixer=sb.SLinOSSMixerConfig(d_state=state, d_head=64, expand=2.0, bc_groups=groups),
                                ffn=sb.SLinOSSMLPConfig(kind=kind, expand=2.0, multiple_of=8, bias=bias))
    return sb.SLinOSSBlock(cfg, device=DEV, dtype=dtype)


# batches at the edges of the 16-row tiles and of the small-batch kernel, more (batch, head) pairs than resident CTAs,
# widths that are no multiple of a warp's run of K or of the output tiles
@pytest.mark.parametrize("batch,d_model,state,groups,kind,bias", [
    (1, 64, 64, None, "swiglu", False), (1, 1024, 128, None, "gelu", True), (3, 200, 64, 1, "swiglu", True),
    (16, 320, 128, 2, "gelu", False), (17, 264, 64, None, "swiglu", False), (33, 128, 128, None, "gelu", True),
    (64, 576, 64, 1, "swiglu", False), (65, 128, 64, None, "gelu", False), (40, 512, 32, None, "swiglu", False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_native_block_step_equals_the_composed_step(batch, d_model, state, groups, kind, bias, dtype, monkeypatch):
    blk = _block(d_model, state, groups, kind, bias, dtype)
    x = torch.randn(4, batch, d_model, device=DEV, dtype=dtype)
    with torch.no_grad():
        native, composed = blk.init_decode_state(batch), blk.init_decode_state(batch)
        got = []
        for t in range(4):
            y, native = blk.step(x[t], native)
            got.append(y)
        monkeypatch.setattr(type(blk), "_native_step", lambda *a: None)
        blk.mixer.decode_backend.fused = False
        want = []
        for t in range(4):
            y, composed = blk.step(x[t], composed)
            want.append(y)
    assert _C.device_status() == 0
    assert rel(torch.stack(got), torch.stack(want)) <= 2e-2
    for a, b in ((native.mixer.scan.state, composed.mixer.scan.state), (native.mixer.conv, composed.mixer.conv),
                 (native.mixer.scan.b_prev, composed.mixer.scan.b_prev), (native.mixer.scan.u_prev, composed.mixer.scan.u_prev)):
        assert a.shape == b.shape and rel(a, b) <= 2e-2


def test_a_decode_token_is_bit_reproducible():
    blk = _block(512, 64, None, "gelu", False, torch.bfloat16)
    x = torch.randn(24, 512, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        runs = []
        for _ in range(2):
            state = blk.init_decode_state(24)
            for _ in range(3):
                y, state = blk.step(x, state)
            runs.append((y, state.mixer.scan.state))
    assert all(torch.equal(a, b) for a, b in zip(*runs))
