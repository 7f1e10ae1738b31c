"""The native decode step of a block (library products and row kernels as one call) and of a mixer (small-batch linear
kernels, pipelined state update) against the composed path: library GEMMs, row kernels, and conv, scan preparation, decode
and tail as launches of their own."""

import copy
import ctypes
import pickle

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


def test_a_token_plan_notices_what_it_relies_on():
    """A replaced or converted parameter, a hook, a swapped child and a copied module all take effect at the next token."""
    blk = _block(128, 64, None, "gelu", True, torch.bfloat16)
    x = torch.randn(3, 128, device=DEV, dtype=torch.bfloat16)

    def token(b):
        with torch.no_grad():
            return b.step(x, b.init_decode_state(3))[0]

    first = token(blk)
    assert torch.equal(token(blk), first) and "_token_plan" in blk.__dict__
    assert torch.equal(token(copy.deepcopy(blk)), first) and torch.equal(token(pickle.loads(pickle.dumps(blk))), first)
    weight = blk.mixer.out_proj.weight
    blk.mixer.out_proj.weight = torch.nn.Parameter(torch.zeros_like(weight))
    assert not torch.equal(token(blk), first)
    blk.mixer.out_proj.weight = weight
    assert torch.equal(token(blk), first)
    calls = []
    handle = blk.ffn.register_forward_hook(lambda *a: calls.append(1))
    assert rel(token(blk), first) <= 2e-2 and calls
    handle.remove()
    ffn, blk.ffn = blk.ffn, _block(128, 64, None, "gelu", True, torch.bfloat16).ffn
    with torch.no_grad():
        blk.ffn.out_proj.bias.add_(1.0)
    assert (token(blk).float() - first.float()).abs().min() > 0.5
    blk.ffn = ffn
    blk.to(torch.float16)
    x = x.to(torch.float16)
    assert rel(token(blk), first) <= 2e-2


@pytest.mark.parametrize("batch", [1, 5, 64, 65])
def test_mixer_token_by_plan_equals_the_composed_token(batch, monkeypatch):
    torch.manual_seed(2)
    mixer = sb.SLinOSSMixer(192, d_state=64, d_head=64, bc_groups=2, device=DEV, dtype=torch.bfloat16)
    x = torch.randn(3, batch, 192, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        a, b, c = (mixer.init_decode_state(batch) for _ in range(3))
        got = [mixer.step(t, a)[0] for t in x]
        monkeypatch.setattr(type(mixer), "_make_token_plan", lambda *a, **k: None)
        mixer.__dict__.pop("_token_plan", None)
        want = [mixer._step(t, b, True, True)[0] for t in x]     # the projections on the library
        plain = [mixer.step(t, c)[0] for t in x]                 # the plan's kernels without the plan
    assert rel(torch.stack(got), torch.stack(want)) <= 1e-2 and rel(a.scan.state, b.scan.state) <= 1e-2
    assert rel(a.scan.b_prev, b.scan.b_prev) <= 1e-2 and rel(a.conv, b.conv) <= 1e-2
    assert all(torch.equal(p, q) for p, q in zip(got, plain)) and torch.equal(a.scan.state, c.scan.state)


@pytest.mark.parametrize("batch, groups", [(1, 1), (24, 1), (64, None)])
def test_a_mixer_token_is_no_farther_from_float64_sums_than_the_composed_one(batch, groups):
    """The same rounding points, and only the sums of the two projections in float64: over the tokens and the whole state the
    small-batch kernels are at most a tenth farther from that than the library's products are."""
    torch.manual_seed(11)
    mixer = sb.SLinOSSMixer(1024, d_state=128, d_head=64, bc_groups=groups, device=DEV, dtype=torch.bfloat16)
    x = torch.randn(24, batch, 1024, device=DEV, dtype=torch.bfloat16)

    def exact(t, state):
        w_in, w_out = mixer.in_proj.weight, mixer.out_proj.weight
        proj = (t.double() @ w_in.double().t()).to(t.dtype)
        gate, value, params, bc = proj.split([mixer.d_inner, mixer.d_inner, mixer.param_proj_dim, mixer.bc_proj_dim], dim=1)
        rows = mixer.decode_backend.fused_step(mixer, gate, value, params, bc, state)
        return (rows.double() @ w_out.double().t()).to(t.dtype), state

    def run(step):
        with torch.no_grad():
            state, out = mixer.init_decode_state(batch), []
            for t in x:
                y, state = step(t, state)
                out += [y.double(), state.scan.state.double(), state.scan.b_prev.double(), state.scan.u_prev.double()]
        return out

    want = run(exact)
    off = [[float((a - b).square().sum() / b.square().sum()) for a, b in zip(run(step), want)]
           for step in (lambda t, s: mixer.step(t, s), lambda t, s: mixer._step(t, s, True, True))]
    for k in range(4):      # y, state, b_prev, u_prev over all tokens
        native, composed = (sum(o[k::4]) ** 0.5 for o in off)
        # either side may have two values more that lie at a tie and round the other way: one bit of bfloat16, 2^-7, of values
        # of the common size each
        ties = (2 / want[k].numel()) ** 0.5 * 2.0 ** -7
        assert native <= 1.1 * composed + ties, (k, native, composed, ties)


# a deep stack multiplies whatever a product's order of sums moves (1.6 % after one token at the last size), so the plan has
# to have the composed path's products, bit for bit
@pytest.mark.parametrize("batch, d_model, dtype, layers, state, groups, kind, tokens", [
    (1, 256, torch.bfloat16, 4, 64, None, "swiglu", 5), (17, 512, torch.float16, 4, 64, None, "swiglu", 5),
    (64, 264, torch.bfloat16, 4, 64, None, "swiglu", 5), (65, 128, torch.bfloat16, 3, 32, 1, "gelu", 3),
    (8, 1024, torch.bfloat16, 6, 128, 1, "swiglu", 20)])
def test_a_stack_token_through_plans_equals_the_composed_token(batch, d_model, dtype, layers, state, groups, kind, tokens, monkeypatch):
    torch.manual_seed(5)
    blk = sb.SLinOSSBlockConfig(d_model=d_model, mixer=sb.SLinOSSMixerConfig(d_state=state, d_head=64, expand=1.0, bc_groups=groups),
                                ffn=sb.SLinOSSMLPConfig(kind=kind, expand=2.0, multiple_of=8, bias=kind == "gelu"))
    stack = sb.SLinOSSStack(sb.SLinOSSStackConfig.uniform(blk, n_layers=layers), device=DEV, dtype=dtype).eval()
    x = torch.randn(tokens, batch, d_model, device=DEV, dtype=dtype)

    def run(step):
        with torch.no_grad():
            state = stack.init_decode_state(batch)
            out = []
            for t in x:
                y, state = step(t, state)
                out.append(y)
        return [torch.stack(out)] + [t for layer in state.layers for t in (layer.mixer.conv, layer.mixer.scan.state,
                                                                          layer.mixer.scan.b_prev, layer.mixer.scan.u_prev)]

    def composed(t, state):    # every product a library call on the weight's own rows
        for b, layer in zip(stack.blocks, state.layers):
            m, carried = b.mixer, layer.mixer
            normed, w = b.mixer_norm(t), m.in_proj.weight
            gate_value, params, bc = (torch.mm(normed, part.t()) for part in w.split(
                [2 * m.d_inner, m.param_proj_dim, m.bc_proj_dim]))
            rows = m.decode_backend.fused_step(m, gate_value[:, :m.d_inner], gate_value[:, m.d_inner:], params, bc, carried)
            t = t + m.out_proj(rows)
            t = t + b.ffn(b.ffn_norm(t))
        return stack.final_norm(t), state

    got = run(stack.step)
    assert all("_token_plan" in b.__dict__ for b in stack.blocks)
    want = run(composed)
    monkeypatch.setattr(sb.SLinOSSBlock, "_make_token_plan", lambda self: None)
    for b in stack.blocks:
        b.__dict__.pop("_token_plan", None)
    plain = run(stack.step)
    assert all("_token_plan" not in b.mixer.__dict__ for b in stack.blocks)
    for a, b, c in zip(got, want, plain):
        assert a.shape == b.shape and torch.equal(a, b) and torch.equal(a, c)


# the projections of the engine's token: either weight of another type than the token, at batches of the small-batch kernel and
# of the library
@pytest.mark.parametrize("batch", [2, 64, 80])
@pytest.mark.parametrize("weights, token", [(torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16),
                                            (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_the_engine_refuses_weights_of_another_type(batch, weights, token):
    from slinoss_b200.engine import MixerDecodeEngine
    mixer = sb.SLinOSSMixer(128, d_state=64, d_head=64, device=DEV, dtype=weights)
    with pytest.raises(RuntimeError, match="dtype"):
        MixerDecodeEngine(mixer, batch, dtype=token)
    mixer.in_proj.to(token)
    with pytest.raises(RuntimeError, match="dtype"):
        MixerDecodeEngine(mixer, batch, dtype=token)
    assert MixerDecodeEngine(mixer.to(token), batch, dtype=token).step(torch.zeros(batch, 128, device=DEV, dtype=token)).isfinite().all()


# the sizes where a block's own products change: row tiles of 16, k tails of 8, biases, parts of in_proj whose width is no
# multiple of 8 (3 heads of 18: that part stays the library's), the longest layers that are the kernel's at 16, 32 and 64 rows
# and the next longer ones (the library's, with the residual sum behind), layers too long for shared memory
@pytest.mark.parametrize("batch, d_model, dtype, d_head, kind, bias, hidden", [
    (1, 8, torch.bfloat16, 8, "gelu", False, 8), (16, 264, torch.float16, 64, "gelu", True, 520),
    (32, 576, torch.bfloat16, 32, "swiglu", True, 1000), (33, 128, torch.float16, 64, "swiglu", False, 72),
    (48, 1024, torch.bfloat16, 64, "gelu", False, 4096), (64, 192, torch.bfloat16, 64, "swiglu", False, 8192),
    (16, 192, torch.float16, 64, "gelu", False, 4096), (16, 192, torch.float16, 64, "gelu", True, 4104),
    (32, 192, torch.bfloat16, 64, "gelu", True, 1536), (32, 192, torch.bfloat16, 64, "gelu", False, 1544),
    (64, 192, torch.bfloat16, 64, "gelu", True, 512), (64, 192, torch.bfloat16, 64, "gelu", False, 520),
    (3, 128, torch.bfloat16, 64, "swiglu", False, 12288)])
def test_token_products_have_the_librarys_bits(batch, d_model, dtype, d_head, kind, bias, hidden, monkeypatch):
    torch.manual_seed(batch)
    blk = sb.SLinOSSBlockConfig(d_model=d_model, mixer=sb.SLinOSSMixerConfig(d_state=64, d_head=d_head, expand=1.0),
                                ffn=sb.SLinOSSMLPConfig(kind=kind, hidden_dim=hidden, multiple_of=8, bias=bias))
    stack = sb.SLinOSSStack(sb.SLinOSSStackConfig.uniform(blk, n_layers=2), device=DEV, dtype=dtype).eval()
    x = torch.randn(3, batch, d_model, device=DEV, dtype=dtype)

    def run():
        with torch.no_grad():
            state, out = stack.init_decode_state(batch), []
            for t in x:
                y, state = stack.step(t, state)
                out.append(y)
        return torch.stack(out)

    got = run()
    planned = ["_token_plan" in b.__dict__ for b in stack.blocks]
    monkeypatch.setattr(sb.SLinOSSBlock, "_make_token_plan", lambda self: None)
    for b in stack.blocks:
        b.__dict__.pop("_token_plan", None)
    assert all(planned) and torch.equal(got, run())


# widths whose products are all the kernel's own, and one with a part left to the library (3 heads of 9) behind 16-row norms
@pytest.mark.parametrize("batch, d_model, by_block", [(4, 512, False), (24, 512, False), (24, 576, False), (4, 512, True)])
def test_a_block_token_overlaps_only_kernels_of_this_library(batch, d_model, by_block):
    """A product that requests its weight ahead of its predecessor's end follows one of this library's kernels: what the program
    queued before the token, and a library product inside it, may write the weight or wait for it.  (Read from the edges of a
    captured token behind an update of the first weight; by_block: in a loop of the program's own, of every block's.)"""
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    def name(node):
        params, = ok(driver.cuGraphKernelNodeGetParams(node))
        got = driver.cuFuncGetName(params.func) if int(params.func) else driver.cuKernelGetName(params.kern)
        return ok(got)[0].decode()

    cfg = sb.SLinOSSBlockConfig(d_model=d_model, mixer=sb.SLinOSSMixerConfig(d_state=64, d_head=64, expand=1.0),
                                ffn=sb.SLinOSSMLPConfig(kind="gelu", expand=2.0, multiple_of=8))
    stack = sb.SLinOSSStack(sb.SLinOSSStackConfig.uniform(cfg, n_layers=2), device=DEV, dtype=torch.bfloat16).eval()
    x = torch.randn(batch, d_model, device=DEV, dtype=torch.bfloat16)

    def token(state):
        if not by_block:
            stack.blocks[0].mixer.in_proj.weight.data.mul_(1.0)
            return stack.step(x, state)
        hidden = x
        for block, carried in zip(stack.blocks, state.layers):
            block.mixer.in_proj.weight.data.mul_(1.0)
            hidden, _ = block.step(hidden, carried)

    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.no_grad():
        state = stack.init_decode_state(batch)
        with torch.cuda.stream(side):
            token(state)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            token(state)
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    edges = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2     # (the binding's edge data does not outlive its call)
    assert edges(raw, None, None, None, ctypes.byref(count)) == 0
    sources, targets, data = (ctypes.c_void_p * count.value)(), (ctypes.c_void_p * count.value)(), (ctypes.c_uint8 * 8 * count.value)()
    assert edges(raw, sources, targets, data, ctypes.byref(count)) == 0
    programmatic = driver.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC.value
    early = [name(driver.CUgraphNode(s)) for s, d in zip(sources, data) if d[2] == programmatic]    # (ports, then the type)
    assert len(early) >= 6 and all(n.startswith("_ZN2sl") for n in early), early


def test_a_dispatch_mode_sees_the_products_of_a_block_token():
    """The plan's products pass the dispatcher by, so under a mode that watches it a block takes the composed path, whose bits the
    plan has."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watch(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(func._schema.name)
            return func(*args, **(kwargs or {}))

    torch.manual_seed(1)
    cfg = sb.SLinOSSBlockConfig(d_model=128, mixer=sb.SLinOSSMixerConfig(d_state=64, d_head=64, expand=1.0),
                                ffn=sb.SLinOSSMLPConfig(kind="gelu", expand=2.0, multiple_of=8))
    stack = sb.SLinOSSStack(sb.SLinOSSStackConfig.uniform(cfg, n_layers=2), device=DEV, dtype=torch.bfloat16).eval()
    x = torch.randn(4, 128, device=DEV, dtype=torch.bfloat16)
    watch = Watch()
    with torch.no_grad():
        want, _ = stack.step(x, stack.init_decode_state(4))
        state = stack.init_decode_state(4)
        with watch:
            got, _ = stack.step(x, state)
    products = [n for n in watch.seen if n in ("aten::mm", "aten::addmm", "aten::linear")]
    assert len(products) >= 2 * 4 and torch.equal(got, want)
