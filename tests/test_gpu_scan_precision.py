"""The float32 scan's gradients against the float64 oracle, closer than the 1e-5 of the parity tests: the products of bfloat16 parts
must not lose what float32 sums token by token keep."""

import pytest
import torch

from oracle import scan_np
from slinoss_b200 import _C
from slinoss_b200.synthetic import make_scan_case
from tests.util import n64, rel

pytestmark = pytest.mark.gpu


# Measured over these very inputs: K 1.25e-7, B 1.37e-7 / 1.28e-7, 1.46e-7; with every product's sum cut off by the tensor cores
# 1.71e-7, 1.88e-7 / 1.51e-7, 1.56e-7.  The bounds lie between.
@pytest.mark.parametrize("T, N, bound_k, bound_b", [(512, 64, 1.45e-7, 1.6e-7), (256, 32, 1.4e-7, 1.51e-7)])
def test_sums_over_the_rows_of_p_are_not_cut_off(T, N, bound_k, bound_b):
    case = make_scan_case(2, 4, T, 64, N, dtype=torch.float32, seed=7)
    c = case.to("cuda")
    grads = _C.scan_bwd(c.U, c.M, c.K, c.B, c.C, None, None, None, c.dY, None, chunk_size=64)
    want = scan_np.v2x2ssd_bwd(*[n64(t) for t in case.tensors()], n64(case.dY))
    assert rel(grads[2], want["K"]) <= bound_k
    assert rel(grads[3], want["B"]) <= bound_b
