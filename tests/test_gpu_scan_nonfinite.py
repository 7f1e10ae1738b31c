"""The float32 scan over operands that are not finite: a NaN or an infinity reaches what depends on it, token by token as in the
recurrence, and nothing else - not the earlier tokens of its chunk, whose products with it are zero."""

import numpy as np
import pytest
import torch

from oracle import scan_np
from slinoss_b200 import _C
from slinoss_b200.synthetic import make_scan_case
from tests.util import n64, rel

pytestmark = pytest.mark.gpu
NAMES = ("U", "M", "K", "B", "C")


# tokens at both ends and inside of the chunks of 16, walked whole (37) and in segments (150); operands of one, two and three parts
@pytest.mark.parametrize("T, token", [(37, 16), (37, 21), (37, 31), (37, 36), (150, 77)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("name, value", [(n, float(v)) for n in ("U", "B", "C", "dY") for v in ("nan", "inf")])
def test_a_value_that_is_not_finite_reaches_what_depends_on_it(name, value, dtype, T, token):
    case = make_scan_case(1, 2, T, 64, 48, dtype=dtype, seed=T, streaming=True, with_init=True)
    getattr(case, name)[0, 1, token, 5] = value
    c = case.to("cuda")
    ops = (c.U, c.M, c.K, c.B, c.C, c.initial_states.float(), c.B_prev, c.U_prev)
    Y, fin = _C.scan_fwd(*ops, chunk_size=64, y_dtype=torch.float32, want_final=True)
    got = dict(zip(NAMES, _C.scan_bwd(*ops, c.dY, None, chunk_size=64)), Y=Y, fin=fin)
    args = [n64(t) for t in case.tensors()]
    kw = dict(initial_states=n64(case.initial_states), B_prev=n64(case.B_prev), U_prev=n64(case.U_prev))
    with np.errstate(all="ignore"):
        wY, wfin, _, _ = scan_np.v2x2ssm(*args, **kw)
        want = dict(scan_np.v2x2ssd_bwd(*args, n64(case.dY), **kw), Y=wY, fin=wfin)
    unit = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]   # one rounding of the result
    for key in ("Y", "fin", "U", "K", "B", "C"):    # (dM comes from sums over all tokens and holds for finite operands)
        g, w = n64(got[key]), want[key]
        finite = np.isfinite(w)
        assert np.isfinite(g[finite]).all(), key
        assert rel(g[finite], w[finite]) <= 1e-5 + (unit if got[key].dtype == dtype else 0.0), key
        if got[key].dtype != torch.float16:         # (float16 results are kept to its finite range)
            assert not np.isfinite(g[~finite]).any(), key


def test_finite_values_above_the_largest_bfloat16():
    """3.395e38 is a float32 that rounds past the largest bfloat16: its row of the output is finite, with the precision of others."""
    case = make_scan_case(1, 1, 40, 64, 16, seed=3)
    case.U[0, 0, 18, 7] = 3.395e38
    c = case.to("cuda")
    Y, _ = _C.scan_fwd(c.U, c.M, c.K, c.B, c.C, None, None, None, chunk_size=64, y_dtype=torch.float32, want_final=False)[:2]
    want = scan_np.v2x2ssm(*[n64(t) for t in case.tensors()])[0]
    rows = np.arange(64) != 7
    assert rel(Y[0, 0, :, 7], want[0, 0, :, 7]) <= 1e-5 and rel(n64(Y)[..., rows], want[..., rows]) <= 1e-5
