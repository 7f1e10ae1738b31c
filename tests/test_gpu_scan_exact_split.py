"""The float32 scan where it is split in time, against the oracle: one segment boundary and many, ragged segments and
token blocks, rows and columns at the edges of the 32-row and 8- and 16-column tiles, several slices of P, carried
state and taps, grouped B/C, a problem large enough to stay whole."""

import pytest
import torch

from oracle import scan_np
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
