"""16-bit scans against the oracle: the tensor-core kernels where they are split in time (segments of one and of several
chunks, a last segment that is shorter, ragged last chunks, carried state and taps, grouped B/C), and widths around the
64 and 128 columns that these hold, which take the float32 sweeps."""

import pytest
import torch

from oracle import scan_np
from slinoss_b200 import _C
from slinoss_b200.ops.v2x2ssd import v2x2ssd
from slinoss_b200.synthetic import make_scan_case
from tests.util import n64, rel

pytestmark = pytest.mark.gpu
NAMES = ("U", "M", "K", "B", "C", "initial_states", "B_prev", "U_prev")


# (batch, heads, groups, T, N, carried state and taps, gradient of the final state)
@pytest.mark.parametrize("shape", [
    (1, 1, 1, 128, 64, False, False), (1, 2, 1, 129, 64, True, True), (1, 1, 1, 1221, 64, True, True),
    (1, 3, 3, 640, 128, True, True), (2, 2, 1, 577, 128, False, True), (1, 2, 2, 200, 4, True, True),
    (1, 2, 2, 333, 32, True, True), (2, 2, 1, 321, 36, False, False), (1, 2, 1, 450, 48, True, True),
    (1, 2, 2, 300, 68, True, True), (1, 2, 2, 260, 96, True, False), (1, 1, 1, 64, 100, False, True),
    (3, 16, 4, 260, 64, True, True), (1, 90, 90, 130, 64, False, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_split_and_padded_scan_matches_the_oracle(shape, dtype):
    b, h, g, T, N, carried, with_dfinal = shape
    case = make_scan_case(b, h, T, 64, N, groups=g, dtype=dtype, seed=T + N, streaming=carried, with_init=carried)
    c = case.to("cuda")
    leaves = {k: getattr(c, k).clone().requires_grad_(True) for k in NAMES if getattr(c, k) is not None}
    Y, fin, _, _ = v2x2ssd(*[leaves[k] for k in "UMKBC"], chunk_size=64, initial_states=leaves.get("initial_states"),
                           B_prev=leaves.get("B_prev"), U_prev=leaves.get("U_prev"))
    d_final = torch.randn(fin.shape, generator=torch.Generator().manual_seed(5)).to(dtype) if with_dfinal else None
    outs, cots = ([Y, fin], [c.dY, d_final.cuda()]) if with_dfinal else ([Y], [c.dY])
    grads = torch.autograd.grad(outs, list(leaves.values()), cots)
    assert _C.device_status() == 0
    args = [n64(t) for t in case.tensors()]
    kw = dict(initial_states=n64(case.initial_states), B_prev=n64(case.B_prev), U_prev=n64(case.U_prev))
    wY, wfin, _, _ = scan_np.v2x2ssm(*args, **kw)
    assert rel(Y, wY) <= 2e-2 and rel(fin, wfin) <= 2e-2
    want = scan_np.v2x2ssd_bwd(*args, n64(case.dY), d_final_state=None if d_final is None else n64(d_final), **kw)
    for name, grad in zip(leaves, grads):
        assert rel(grad, want[name]) <= 2e-2, (name, rel(grad, want[name]))


@pytest.mark.parametrize("N", [64, 128])
def test_forward_without_its_workspace_walks_whole_or_is_refused(N):
    c = make_scan_case(1, 2, 1300, 64, N, dtype=torch.bfloat16, seed=N).to("cuda")
    assert _C.workspace_bytes(_C.WS_SCAN_FWD, 1, 2, 2, 1300, 64, N, 64, torch.bfloat16) > 0
    want, _ = _C.scan_fwd(c.U, c.M, c.K, c.B, c.C, None, None, None, chunk_size=64, y_dtype=torch.float32, want_final=False)
    Y = torch.full_like(want, float("nan"))
    status = _C.lib().sl_v2x2ssd_fwd(*[t.data_ptr() for t in (c.U, c.M, c.K, c.B, c.C)], None, None, None, Y.data_ptr(), None, None,
                                     1, 2, 2, 1300, 64, N, 64, _C.SL_BF16, _C.SL_F32, _C.PATH_AUTO, None, 0,
                                     torch.cuda.current_stream().cuda_stream)
    if N == 128:
        assert _C.lib().sl_status_string(status).decode() == "workspace missing or too small"
    else:
        assert status == 0 and rel(Y, want) <= 2e-2 and _C.device_status() == 0


# Reverse sweeps whose last round of CTAs gives the ends of its streams to idle SMs: no whole stream and some, a tail of one
# chunk (ragged) and of several, two column blocks, grouped B/C, carried state and taps.  Against the float32 sweeps on the
# same 16-bit operands, which are held to the oracle elsewhere: the bar of 16-bit scans.
@pytest.mark.parametrize("b, h, g, T, N, carried, with_dfinal", [
    (8, 16, 16, 2500, 64, False, True), (4, 32, 4, 2111, 64, True, True), (8, 32, 32, 2049, 64, False, False),
    (4, 16, 16, 2305, 128, True, False), (10, 10, 10, 2177, 64, True, True)])
def test_streams_that_give_their_end_to_idle_sms(b, h, g, T, N, carried, with_dfinal):
    c = make_scan_case(b, h, T, 64, N, groups=g, dtype=torch.bfloat16, seed=T, streaming=carried, with_init=carried).to("cuda")
    z0 = None if c.initial_states is None else c.initial_states.float()
    ops = (c.U, c.M, c.K, c.B, c.C, z0, c.B_prev, c.U_prev)
    d_final = torch.randn(b, h, 64, 2 * N, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) if with_dfinal else None
    got = _C.scan_bwd(*ops, c.dY, d_final, chunk_size=64)
    want = _C.scan_bwd(*ops, c.dY, d_final, chunk_size=64, path="simt")
    assert _C.device_status() == 0
    for name, x, y in zip(NAMES, got, want):
        assert (x is None) == (y is None)
        if x is not None:
            assert rel(x, y) <= 2e-2, (name, rel(x, y))
