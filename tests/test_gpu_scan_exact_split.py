"""The float32 scan where it is split in time, against the oracle: one segment boundary and many, ragged segments and
token blocks, rows and columns at the edges of the 32-row and 8- and 16-column tiles, several slices of P, carried
state and taps, grouped B/C, a problem large enough to stay whole."""

import pytest
import torch

from oracle import scan_np
from slinoss_b200 import _C
from slinoss_b200.ops.v2x2ssd import v2x2ssd
from slinoss_b200.synthetic import make_scan_case
from tests.util import n64, rel

pytestmark = pytest.mark.gpu
NAMES = ("U", "M", "K", "B", "C", "initial_states", "B_prev", "U_prev")


# (batch, heads, groups, T, P, N, carried state and taps, gradient of the final state)
@pytest.mark.parametrize("shape", [
    (1, 1, 1, 65, 64, 32, True, True), (1, 2, 1, 80, 33, 8, False, True), (2, 2, 2, 97, 32, 9, True, False),
    (1, 2, 2, 256, 64, 33, True, True), (1, 1, 1, 300, 70, 1, True, True), (1, 1, 1, 513, 1, 128, False, True),
    (1, 2, 1, 1030, 65, 7, True, True), (2, 1, 1, 64, 64, 32, True, True), (8, 40, 40, 70, 64, 5, False, True)])
def test_split_float32_scan_matches_the_oracle(shape):
    b, h, g, T, P, N, carried, with_dfinal = shape
    case = make_scan_case(b, h, T, P, N, groups=g, dtype=torch.float32, seed=T + N, streaming=carried, with_init=carried)
    c = case.to("cuda")
    leaves = {k: getattr(c, k).clone().requires_grad_(True) for k in NAMES if getattr(c, k) is not None}
    Y, fin, _, _ = v2x2ssd(*[leaves[k] for k in "UMKBC"], chunk_size=64, initial_states=leaves.get("initial_states"),
                           B_prev=leaves.get("B_prev"), U_prev=leaves.get("U_prev"))
    d_final = torch.randn(fin.shape, generator=torch.Generator().manual_seed(5)) if with_dfinal else None
    outs, cots = ([Y, fin], [c.dY, d_final.cuda()]) if with_dfinal else ([Y], [c.dY])
    grads = torch.autograd.grad(outs, list(leaves.values()), cots)
    args = [n64(t) for t in case.tensors()]
    kw = dict(initial_states=n64(case.initial_states), B_prev=n64(case.B_prev), U_prev=n64(case.U_prev))
    wY, wfin, _, _ = scan_np.v2x2ssm(*args, **kw)
    assert rel(Y, wY) <= 1e-5 and rel(fin, wfin) <= 1e-5
    want = scan_np.v2x2ssd_bwd(*args, n64(case.dY), d_final_state=None if d_final is None else n64(d_final), **kw)
    for name, grad in zip(leaves, grads):
        assert rel(grad, want[name]) <= 1e-5, (name, rel(grad, want[name]))


# 16-bit operands of widths that the tensor-core kernels do not hold take the float32 sweeps: the operands are exact, so
# float32 results keep the float32 bar and 16-bit ones add one rounding; a zero transition (a forgotten past) is computed
# through, where the chunked kernels would divide by it
@pytest.mark.parametrize("dtype, unit", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11)])
@pytest.mark.parametrize("N, groups, T", [(4, 2, 70), (32, 1, 257), (48, 2, 333), (60, 2, 64), (68, 1, 130), (124, 2, 200)])
def test_16_bit_operands_of_other_widths_keep_float32_precision(N, groups, T, dtype, unit):
    case = make_scan_case(1, 2, T, 64, N, groups=groups, dtype=dtype, seed=T + N, streaming=True, with_init=True)
    zero = T // 3
    case.M[:, 1, zero] = 0.0
    c = case.to("cuda")
    ops = (c.U, c.M, c.K, c.B, c.C, c.initial_states.float(), c.B_prev, c.U_prev)
    Y, fin, states = _C.scan_fwd(*ops, chunk_size=64, y_dtype=torch.float32, want_final=True, save_states=True)
    got = _C.scan_bwd(*ops, c.dY, None, chunk_size=64)
    assert states is None
    with pytest.raises(RuntimeError):
        _C.scan_fwd(*ops, chunk_size=64, y_dtype=dtype, want_final=False, path="tc")
    args = [n64(t) for t in case.tensors()]
    kw = dict(initial_states=n64(case.initial_states), B_prev=n64(case.B_prev), U_prev=n64(case.U_prev))
    wY, wfin, _, _ = scan_np.v2x2ssm(*args, **kw)
    assert rel(Y, wY) <= 1e-5 and rel(fin, wfin) <= 1e-5
    want = scan_np.v2x2ssd_bwd(*args, n64(case.dY), **kw)
    want["M"][:, 1, zero] = 0.0    # (not defined by the formula S / conj(m) that the sweeps use)
    for name, grad in zip(NAMES, got):
        if name in ("initial_states", "M", "K"):
            assert grad.dtype == torch.float32 and rel(grad, want[name]) <= 1e-5, (name, rel(grad, want[name]))
        else:
            assert grad.dtype == dtype and rel(grad, want[name]) <= unit + 1e-5, (name, rel(grad, want[name]))


# Edges of the chunks of 16 tokens, of the warps of 16 columns, of the slices of 64 rows and of the 16-byte pieces in which
# rows are staged, each operand type beside each type of dY (the products are of one, two or three bfloat16 parts of it).
# Operands are exact in every case, and sums of 24-bit products err by 2^-24 of their terms: the float32 bar holds.
@pytest.mark.parametrize("dtype, dy_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16),
                                             (torch.bfloat16, torch.float32), (torch.float16, torch.bfloat16),
                                             (torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("b, h, g, T, P, N", [(1, 2, 1, 1, 64, 16), (2, 1, 1, 15, 1, 17), (1, 2, 2, 16, 63, 15),
                                              (1, 1, 1, 17, 65, 48), (1, 3, 1, 33, 130, 31), (1, 2, 2, 97, 64, 128),
                                              (1, 1, 1, 1500, 9, 1), (1, 1, 1, 1041, 64, 65)])
def test_chunks_of_bfloat16_parts_at_their_edges(b, h, g, T, P, N, dtype, dy_dtype):
    case = make_scan_case(b, h, T, P, N, groups=g, dtype=dtype, seed=T + 3 * N, streaming=True, with_init=True)
    gen = torch.Generator().manual_seed(T)
    dY = torch.randn(b, h, T, P, generator=gen).to(dy_dtype)
    d_final = torch.randn(b, h, P, 2 * N, generator=gen)
    c = case.to("cuda")
    ops = (c.U, c.M, c.K, c.B, c.C, c.initial_states.float(), c.B_prev, c.U_prev)
    Y, fin = _C.scan_fwd(*ops, chunk_size=64, y_dtype=torch.float32, want_final=True, path="simt")
    got = _C.scan_bwd(*ops, dY.cuda(), d_final.cuda(), chunk_size=64, path="simt")
    args = [n64(t) for t in case.tensors()]
    kw = dict(initial_states=n64(case.initial_states), B_prev=n64(case.B_prev), U_prev=n64(case.U_prev))
    wY, wfin, _, _ = scan_np.v2x2ssm(*args, **kw)
    assert rel(Y, wY) <= 1e-5 and rel(fin, wfin) <= 1e-5
    want = scan_np.v2x2ssd_bwd(*args, n64(dY), d_final_state=n64(d_final), **kw)
    unit = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]   # one rounding of the result
    for name, grad in zip(NAMES, got):
        bar = 1e-5 + (unit if grad.dtype == dtype else 0.0)
        assert rel(grad, want[name]) <= bar, (name, rel(grad, want[name]))
