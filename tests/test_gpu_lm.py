"""The stacked-LM training step on one GPU: its shortcuts (clipping folded into the fused optimizer,
the head GEMM without the last position, the projection's own backward pass) against the plain
formulation of the same step."""

import copy

import pytest
import torch
import torch.nn.functional as F

from slinoss_b200.lm import DataParallelTrainer, SLinOSSLM, lm_stack_config
from slinoss_b200.ops.mixer import split_mixer_projection
from tests.util import rel

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(dtype=torch.float32):
    torch.manual_seed(0)
    return SLinOSSLM(512, lm_stack_config(256, 2), device=DEV, dtype=dtype)


def test_loss_drops_the_last_position_before_the_head():
    m = _model()
    ids = torch.randint(0, 512, (2, 96), device=DEV)
    logits = m(ids)
    want = F.cross_entropy(logits[:, :-1].reshape(-1, 512).float(), ids[:, 1:].reshape(-1))
    assert rel(m.loss(ids), want) <= 1e-6


@pytest.mark.parametrize("clip", [1e-3, 1e3])        # one that clips, one that does not
def test_clipping_inside_the_fused_optimizer_equals_clip_then_step(clip):
    a = _model()
    b = copy.deepcopy(a)
    ids = torch.randint(0, 512, (2, 128), device=DEV)
    ta = DataParallelTrainer(a, grad_clip=clip, reduce=False)
    tb = DataParallelTrainer(b, grad_clip=0.0, reduce=False)
    for _ in range(2):
        ta.step(ids)
        # the plain formulation: scale the gradients, then step
        tb.opt.zero_grad(set_to_none=True)
        b.loss(ids).backward()
        norm = torch.nn.utils.clip_grad_norm_(b.parameters(), clip)
        tb.opt.step()
        assert rel(ta.last_grad_norm, norm) <= 1e-5
    for (n, pa), pb in zip(a.named_parameters(), b.parameters()):
        assert rel(pa, pb) <= 1e-5, n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_projection_backward_equals_autograd_of_the_three_gemms(dtype):
    torch.manual_seed(1)
    x = torch.randn(3, 50, 128, device=DEV).to(dtype).requires_grad_()
    w = (0.1 * torch.randn(2 * 96 + 12 + 64, 128, device=DEV)).to(dtype).requires_grad_()
    outs = split_mixer_projection(x, w, d_inner=96, param_proj_dim=12)
    gs = [torch.randn_like(o) for o in outs]
    torch.autograd.backward(outs, gs)
    x2, w2 = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    full = F.linear(x2, w2)
    want = torch.split(full, [96, 96, 12, 64], dim=-1)
    torch.autograd.backward(want, [g.double() for g in gs])
    t = 1e-5 if dtype == torch.float32 else 2e-2
    for o, o2 in zip(outs, want):
        assert rel(o, o2) <= t
    assert rel(x.grad, x2.grad) <= t and rel(w.grad, w2.grad) <= t


@pytest.mark.parametrize("rows,vocab", [(1, 1), (3, 7), (5, 256), (17, 4099), (9, 32000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cross_entropy_and_its_gradient_equal_torch(rows, vocab, dtype):
    from slinoss_b200.lm import cross_entropy
    torch.manual_seed(rows)
    logits = (4 * torch.randn(rows, vocab, device=DEV)).to(dtype).requires_grad_()
    targets = torch.randint(0, vocab, (rows,), device=DEV)
    want_in = logits.detach().double().requires_grad_()
    for reduction in ("mean", "sum"):
        loss, want = cross_entropy(logits, targets, reduction=reduction), F.cross_entropy(want_in, targets, reduction=reduction)
        (g,), (gw,) = torch.autograd.grad(loss * 3, logits), torch.autograd.grad(want * 3, want_in)
        t = 1e-5 if dtype == torch.float32 else 1e-2
        assert rel(loss, want) <= 1e-5 and (rel(g, gw) <= t or (g - gw).abs().max() < 1e-6)


@pytest.mark.parametrize("rows,vocab,ignored", [(1, 7, 1), (5, 256, 2), (1030, 33, 1029), (2, 4099, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cross_entropy_leaves_out_the_ignored_index(rows, vocab, ignored, dtype):
    from slinoss_b200.lm import cross_entropy
    torch.manual_seed(rows)
    logits = (4 * torch.randn(rows, vocab, device=DEV)).to(dtype).requires_grad_()
    targets = torch.randint(0, vocab, (rows,), device=DEV)
    targets[torch.randperm(rows, device=DEV)[:ignored]] = -100
    want_in = logits.detach().double().requires_grad_()
    for reduction in ("mean", "sum", "none"):
        loss, want = cross_entropy(logits, targets, reduction=reduction), F.cross_entropy(want_in, targets, reduction=reduction)
        assert loss.shape == want.shape
        if rows == ignored and reduction == "mean":
            assert loss.isnan() and want.isnan()
            continue
        (g,), (gw,) = torch.autograd.grad(loss.sum(), logits), torch.autograd.grad(want.sum(), want_in)
        t = 1e-5 if dtype == torch.float32 else 1e-2
        assert rel(loss, want) <= 1e-5 and rel(g, gw) <= t
        assert g[targets == -100].count_nonzero() == 0


@pytest.mark.parametrize("n,vocab,width", [(1, 1, 8), (40, 7, 12), (300, 1000, 264), (513, 33, 2048)])
def test_embedding_gradient_equals_torch(n, vocab, width):
    from slinoss_b200.lm import embed
    table = torch.nn.Embedding(vocab, width, device=DEV, dtype=torch.bfloat16)
    ids = torch.randint(0, vocab, (n,), device=DEV)
    d = torch.randn(n, width, device=DEV, dtype=torch.bfloat16)
    (g,) = torch.autograd.grad(embed(ids, table), table.weight, d)
    want = torch.zeros(vocab, width, device=DEV, dtype=torch.float64).index_add_(0, ids, d.double())
    assert rel(g, want) <= 5e-3


@pytest.mark.parametrize("betas", [(0.9, 0.999), (0.9, 0.95), (0.0, 0.9999)])
def test_adamw_keeps_float32_precision_for_betas_near_one(betas):
    """From zero parameters a step is the update itself: a few float32 roundings (2^-24 each) from float64, in the states too."""
    from slinoss_b200.optim import AdamW
    torch.manual_seed(3)
    p = torch.nn.Parameter(torch.zeros(4096, device=DEV))
    q = torch.nn.Parameter(torch.zeros(4096, dtype=torch.float64))
    kw = dict(lr=1e-3, betas=betas, eps=1e-8, weight_decay=0.05)
    a, b = AdamW([p], **kw), torch.optim.AdamW([q], **kw)
    for _ in range(4):
        p.grad = torch.rand_like(p) + 0.5
        q.grad = p.grad.double().cpu()
        a.step()
        b.step()
        sa, sb = a.state[p], b.state[q]
        for got, want in ((p, q), (sa["exp_avg"], sb["exp_avg"]), (sa["exp_avg_sq"], sb["exp_avg_sq"])):
            assert float(((got.detach().double().cpu() - want.detach()) / want.detach()).abs().max()) <= 12 * 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_adamw_equals_torch_also_after_loading_its_state_and_with_missing_gradients(dtype):
    from slinoss_b200.optim import AdamW
    torch.manual_seed(2)
    shapes = [(1,), (7, 3), (64, 129), (8193,), (300, 256)] + [(5,)] * 70
    a = [torch.nn.Parameter(torch.randn(s, device=DEV).to(dtype)) for s in shapes]
    b = [torch.nn.Parameter(p.detach().clone()) for p in a]
    groups = lambda ps: [{"params": ps[:3], "weight_decay": 0.05}, {"params": ps[3:], "weight_decay": 0.0}]
    oa = AdamW(groups(a), lr=1e-2, betas=(0.9, 0.95))
    ob = torch.optim.AdamW(groups(b), lr=1e-2, betas=(0.9, 0.95), fused=True)
    for it in range(6):
        for i, (p, q) in enumerate(zip(a, b)):
            p.grad = None if (it == 3 and i % 2) else torch.randn_like(p)
            q.grad = None if p.grad is None else p.grad.clone()
        if it == 4:
            state = oa.state_dict()
            oa.load_state_dict(copy.deepcopy(ob.state_dict()))
            ob.load_state_dict(copy.deepcopy(state))
        oa.step()
        ob.step()
        for p, q in zip(a, b):
            # (in bfloat16 a state may round the other way, which moves an element by a part of a step)
            assert float((p - q).detach().abs().max()) <= (1e-5 if dtype == torch.float32 else 2e-2), (it, tuple(p.shape))
            assert p.grad is None or torch.equal(p.grad, q.grad)
            assert (p in oa.state) == (q in ob.state) and float(oa.state[p]["step"]) == float(ob.state[q]["step"])
