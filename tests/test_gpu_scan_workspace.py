"""The float32 backward inside exactly the workspace that it asks for, walked whole and in segments, with B and C of every head's
own (no scratch per head), shared, and over two slices of P (sums in the scratch)."""

import pytest
import torch

from slinoss_b200 import _C
from slinoss_b200.synthetic import make_scan_case
from tests.util import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch, heads, groups, T, P, N", [(2, 2, 2, 70, 64, 20), (1, 4, 2, 200, 64, 48), (1, 2, 2, 100, 80, 32),
                                                           (1, 2, 1, 1, 64, 8)])
@pytest.mark.parametrize("split", [False, True])
def test_the_backward_stays_inside_its_workspace(batch, heads, groups, T, P, N, split):
    c = make_scan_case(batch, heads, T, P, N, groups=groups, seed=T, streaming=True, with_init=True).to("cuda")
    args = (c.U, c.M, c.K, c.B, c.C, c.initial_states, c.B_prev, c.U_prev)
    want = _C.scan_bwd(*args, c.dY, None, chunk_size=64, path="simt")
    bh, shared = batch * heads, groups != heads or P > 64
    whole = (4 * (2 * bh * (T + 1) + (4 * bh * T * N + 2 * bh * N if shared else 0)) + 255) // 256 * 256
    asked = _C.workspace_bytes(_C.WS_SCAN_BWD, batch, heads, groups, T, P, N, 64, torch.float32, "simt")
    assert asked == whole if T <= 64 else asked > whole
    n = asked if split else whole
    room = torch.full((n + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
    outs = [torch.full_like(w, float("nan")) for w in want]
    ptr = lambda t: t.data_ptr()
    status = _C.lib().sl_v2x2ssd_bwd(*map(ptr, args), None, None, ptr(c.dY), None, *map(ptr, outs), batch, heads, groups, T, P, N, 64,
                                     _C.SL_F32, _C.SL_F32, _C.PATH_SIMT, ptr(room), n, torch.cuda.current_stream().cuda_stream)
    assert status == 0 and bool((room[n:] == 0xA5).all())
    for got, ref in zip(outs, want):
        assert rel(got, ref) <= 1e-5      # (whole and split walks round differently)
