"""The whole-mixer native path against the stage-by-stage path of the same module (conv + preparation, scan, tail and
projections as separate ops), where its layout can go wrong: head counts that leave the bc columns unaligned, odd
lengths, one and several groups, state sizes on both sides of the wide B/C kernels, scalar head sizes, every conv width."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 2e-4, torch.bfloat16: 3e-2, torch.float16: 6e-3}


def _mixer(d_model, d_state, d_head, groups, d_conv, dtype):
    from slinoss_b200 import SLinOSSMixer
    torch.manual_seed(7)
    return SLinOSSMixer(d_model, d_state=d_state, expand=2, d_head=d_head, d_conv=d_conv, bc_groups=groups,
                        device="cuda", dtype=dtype)


def _close(a, b, tol, name):
    scale = b.float().abs().max().clamp_min(1e-6)
    assert ((a.float() - b.float()).abs().max() / scale).item() < tol, name


@pytest.mark.parametrize("d_model, d_state, d_head, groups, d_conv, batch, T, dtype", [
    (128, 64, 64, None, 4, 2, 130, torch.bfloat16),      # 3H = 12: bc starts past a gap
    (512, 64, 64, 4, 4, 1, 64, torch.bfloat16),          # 3H = 48: one GEMM
    (288, 128, 64, 1, 4, 2, 197, torch.bfloat16),        # wide B/C rows, one group, 9 heads
    (256, 96, 64, 8, 3, 1, 65, torch.float16),
    (64, 68, 64, 1, 2, 1, 3, torch.bfloat16),
    (96, 20, 32, 3, 1, 2, 33, torch.float16),
    (30, 6, 5, None, 4, 2, 17, torch.float32),           # nothing aligned
    (128, 32, 64, 2, 4, 3, 100, torch.float32),
])
def test_native_mixer_matches_stages(monkeypatch, d_model, d_state, d_head, groups, d_conv, batch, T, dtype):
    m = _mixer(d_model, d_state, d_head, groups, d_conv, dtype)
    x = torch.randn(batch, T, d_model, device="cuda").to(dtype)
    dy = torch.randn(batch, T, d_model, device="cuda").to(dtype)
    tol = TOL[dtype]

    def run():
        m.zero_grad(set_to_none=True)
        xi = x.clone().requires_grad_()
        y = m(xi)
        y.backward(dy)
        with torch.no_grad():
            h = max(T // 2, 1)
            y0, st = m(x[:, :h], return_state=True)
            y1, st = m(x[:, h:], state=st, return_state=True) if h < T else (y0[:, :0], st)
        outs = {"y": y.detach(), "dx": xi.grad, "y0": y0, "y1": y1, "conv": st.conv, "state": st.scan.state,
                "b_prev": st.scan.b_prev, "u_prev": st.scan.u_prev}
        outs.update({n: p.grad for n, p in m.named_parameters()})
        return outs

    got = run()
    monkeypatch.setattr(type(m), "_native_forward_ready", lambda self, x, state: False)
    want = run()
    assert got.keys() == want.keys()
    for name, ref in want.items():
        assert got[name].shape == ref.shape and got[name].dtype == ref.dtype, name
        if ref.numel():
            _close(got[name], ref, tol, name)
