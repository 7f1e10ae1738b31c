"""The work that users of this framework have it do, as timed cases.

Every case is one pass through a public entry point, over the range of sizes, types and options that the
configurations, the tests and the benchmark of this repository use:

``scan_train``     ``v2x2ssd_cute`` forward + ``torch.autograd.grad``: the scan operator inside a training loop
``scan_prefill``   ``v2x2ssd`` on a prompt segment with the carried state in and out, no gradients
``scan_decode``    ``v2x2ssd_decode``: one token over the carried float32 state, updated in place
``mixer_train``    ``SLinOSSMixer`` forward + backward: gradients of the input and of every parameter
``mixer_prefill``  ``SLinOSSMixer.forward(return_state=True)`` without gradients: a prompt before decoding
``mixer_step``     ``SLinOSSMixer.step``: one eager decode token, state in place
``engine_step``    ``MixerDecodeEngine.step``: one decode token of the CUDA-graph engine
``stack_step``     ``SLinOSSStack.step``: one eager decode token of a whole stack of blocks
``lm_train``       ``DataParallelTrainer.step`` of a ``SLinOSSLM`` on one GPU: forward, backward, clipping, AdamW

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a program
has in hand before the call (inputs, modules, carried state), ``run`` is the call, ``work`` what it cannot do
without, ``tolerance`` how far two correct implementations at the same precision may differ.
"""

import math

import torch

import slinoss_b200 as sb
from slinoss_b200.engine import MixerDecodeEngine
from slinoss_b200.lm import DataParallelTrainer, SLinOSSLM
from slinoss_b200.ops.v2x2ssd import v2x2ssd, v2x2ssd_cute, v2x2ssd_decode
from slinoss_b200.synthetic import foh_taps_from_polar

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
P = 64       # head dimension of every configuration
CHUNK = 64   # and their chunk size


def _scan(name, kind, batch, heads, groups, seq, state, dtype, carried=False):
    return {"name": name, "kind": kind, "batch": batch, "heads": heads, "groups": groups, "seq": seq,
            "state": state, "dtype": dtype, "carried": carried}


def _mixer(name, kind, batch, seq, d_model, groups, state, dtype):
    """``groups`` 0: one B/C group per head; ``seq`` 1 for the decode kinds."""
    return {"name": name, "kind": kind, "batch": batch, "seq": seq, "d_model": d_model, "groups": groups,
            "state": state, "dtype": dtype}


def listed():
    return [
        # the headline: scan forward + backward at the benchmark's size
        _scan("scan_train_bench", "scan_train", 8, 16, 16, 4096, 64, "bf16"),
        # the default shape of the scan benchmark this operator is compared on: 48 oscillators, half precision
        _scan("scan_train_48_fp16", "scan_train", 16, 4, 4, 2048, 48, "fp16"),
        # the reference-sized float32 problem: the smallest training call
        _scan("scan_train_small_fp32", "scan_train", 2, 4, 4, 256, 32, "fp32"),
        # one long prompt, continued from a carried state: few streams, many tokens, a ragged end
        _scan("scan_prefill_long", "scan_prefill", 1, 16, 16, 16383, 64, "bf16", True),
        # one token for a large serving batch at the decode configuration: bound by the float32 state
        _scan("scan_decode_batch", "scan_decode", 256, 32, 32, 1, 64, "bf16"),
        # one mixer layer in training at the mixer configuration
        _mixer("mixer_train_bench", "mixer_train", 8, 2048, 1024, 0, 64, "bf16"),
        # a prompt of odd length through one mixer with the default 128 oscillators
        _mixer("mixer_prefill_odd", "mixer_prefill", 1, 1021, 1024, 0, 128, "bf16"),
        # interactive decoding, one sequence, eager: the smallest serving call
        _mixer("mixer_step_single", "mixer_step", 1, 1, 1024, 0, 128, "bf16"),
        # the graph engine at the decode configuration's batch
        _mixer("engine_step_batch", "engine_step", 256, 1, 1024, 0, 64, "bf16"),
        # one token through a stack of blocks for a small serving batch
        {"name": "stack_step_small", "kind": "stack_step", "batch": 8, "d_model": 512, "layers": 4, "groups": 1,
         "state": 128, "ffn": "swiglu", "dtype": "bf16"},
        # the training model of the reference's harness (width 576, shared B/C, GELU x4 with bias), three blocks
        {"name": "lm_train_narrow", "kind": "lm_train", "batch": 4, "seq": 2048, "d_model": 576, "layers": 3,
         "expand": 2.0, "groups": 1, "state": 128, "vocab": 256, "bias": True, "dtype": "bf16"},
        # the stacked-LM configuration (width 2048, 32 heads, vocabulary 32000), two of its blocks: the largest call
        {"name": "lm_train_wide", "kind": "lm_train", "batch": 4, "seq": 4096, "d_model": 2048, "layers": 2,
         "expand": 1.0, "groups": 0, "state": 64, "vocab": 32000, "bias": False, "dtype": "bf16"},
    ]


# ---- further cases of the same ranges ---------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _groups_of(rng, heads):
    return rng.choice([g for g in range(1, heads + 1) if heads % g == 0] + [heads] * 3)


def draw(rng):
    kind = rng.choice(["scan_train", "scan_train", "scan_prefill", "scan_decode", "mixer_train", "mixer_prefill",
                       "mixer_step", "engine_step", "stack_step", "lm_train"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "scan_train":
        dtype = rng.choice([half, half, half, "fp32"])
        tokens = 1 << 19 if dtype != "fp32" else 1 << 15     # batch * heads * seq
        batch, heads = _log_int(rng, 1, 16), _log_int(rng, 1, 32)
        seq = _log_int(rng, 100, max(200, min(8192, tokens // (batch * heads))))
        return {"kind": kind, "batch": batch, "heads": heads, "groups": _groups_of(rng, heads), "seq": seq,
                "state": rng.choice([32, 48, 64, 64, 128, 128] if dtype != "fp32" else [32, 48, 64]), "dtype": dtype,
                "carried": rng.random() < 0.25}
    if kind == "scan_prefill":
        batch, heads = _log_int(rng, 1, 8), rng.choice([8, 16, 18, 32, 64])
        return {"kind": kind, "batch": batch, "heads": heads, "groups": _groups_of(rng, heads),
                "seq": _log_int(rng, 64, max(256, min(32768, (1 << 20) // (batch * heads)))),
                "state": rng.choice([64, 128]), "dtype": half, "carried": rng.random() < 0.75}
    if kind == "scan_decode":
        heads, state = rng.choice([8, 16, 18, 32, 64]), rng.choice([32, 48, 64, 128])
        return {"kind": kind, "batch": _log_int(rng, 1, min(512, 256 * 32 * 64 // (heads * state))), "heads": heads,
                "groups": _groups_of(rng, heads), "seq": 1, "state": state, "dtype": rng.choice([half, half, "fp32"]),
                "carried": False}
    if kind in ("mixer_train", "mixer_prefill"):
        d_model = 64 * rng.randint(4, 16)
        batch = _log_int(rng, 1, 8)
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 64, min(4096, 16384 // batch)), "d_model": d_model,
                "groups": rng.choice([0, 0, 1, 2]), "state": rng.choice([64, 128]), "dtype": half}
    if kind in ("mixer_step", "engine_step"):
        return {"kind": kind, "batch": _log_int(rng, 1, 256), "seq": 1, "d_model": 64 * rng.randint(4, 16),
                "groups": rng.choice([0, 0, 1, 2]), "state": rng.choice([64, 128]), "dtype": half}
    if kind == "stack_step":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "d_model": 64 * rng.randint(4, 16),
                "layers": rng.randint(2, 6), "groups": rng.choice([0, 1]), "state": rng.choice([64, 128]),
                "ffn": rng.choice(["swiglu", "gelu"]), "dtype": "bf16"}
    batch = _log_int(rng, 1, 8)
    return {"kind": kind, "batch": batch, "seq": _log_int(rng, 128, 8192 // batch), "d_model": 64 * rng.randint(4, 16),
            "layers": rng.randint(1, 3), "expand": rng.choice([1.0, 2.0]), "groups": rng.choice([0, 1]),
            "state": rng.choice([64, 128]), "vocab": rng.choice([256, 8000, 32000]), "bias": rng.random() < 0.5,
            "dtype": "bf16"}


# ---- preparation ------------------------------------------------------------------------------------------
def _scan_inputs(case, gen):
    """The value distributions of the scan configurations: damping radius in [0.9, 0.999], uniform angle, exact
    first-order-hold taps, B and C with standard deviation 1/sqrt(N)."""
    b, h, g, T, N = case["batch"], case["heads"], case["groups"], case["seq"], case["state"]
    io = DTYPES[case["dtype"]]
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    r = torch.exp(-torch.nn.functional.softplus(rn(b, h, T))).clamp(0.9, 0.999)
    theta = (torch.rand(b, h, T, generator=gen, device="cuda") * 2 - 1) * math.pi
    dt = 5e-3 + (1e-1 - 5e-3) * torch.sigmoid(rn(b, h, T))
    out = {"U": rn(b, h, T, P).to(io),
           "M": torch.stack((r * torch.cos(theta), r * torch.sin(theta)), dim=-1).contiguous(),
           "K": foh_taps_from_polar(dt, r, theta).contiguous(),
           "B": (rn(b, g, T, 2 * N) / math.sqrt(N)).to(io), "C": (rn(b, g, T, 2 * N) / math.sqrt(N)).to(io)}
    if case["carried"]:
        out["initial_states"] = 0.1 * rn(b, h, P, 2 * N)
        out["B_prev"] = (rn(b, g, 2 * N) / math.sqrt(N)).to(io)
        out["U_prev"] = rn(b, h, P).to(io)
    return out, rn


def _init_linear(module, gen):
    with torch.no_grad():
        for m in module.modules():
            if isinstance(m, torch.nn.Linear):
                m.weight.normal_(0.0, 0.02, generator=gen)
                if m.bias is not None:
                    m.bias.normal_(0.0, 0.02, generator=gen)


def _mixer_config(case):
    return sb.SLinOSSMixerConfig(d_state=case["state"], d_head=P, d_conv=4, chunk_size=CHUNK,
                                 expand=case.get("expand", 2.0), bc_groups=case["groups"] or None)


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    io = DTYPES[case["dtype"]]
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(io)
    if kind == "scan_train":
        ins, rn32 = _scan_inputs(case, gen)
        return {"kind": kind, "inputs": {k: t.requires_grad_(True) for k, t in ins.items()},
                "dY": rn32(*ins["U"].shape).to(io)}
    if kind == "scan_prefill":
        return {"kind": kind, "inputs": _scan_inputs(case, gen)[0]}
    if kind == "scan_decode":
        ins, rn32 = _scan_inputs(case, gen)
        b, h, g, N = case["batch"], case["heads"], case["groups"], case["state"]
        return {"kind": kind, "token": [ins[k][:, :, 0].contiguous() for k in "UMKBC"],
                "state": 0.1 * rn32(b, h, P, 2 * N), "B_prev": (rn32(b, g, 2 * N) / math.sqrt(N)).to(io),
                "U_prev": rn32(b, h, P).to(io)}
    if kind == "lm_train":
        d = case["d_model"]
        block = sb.SLinOSSBlockConfig(
            d_model=d, mixer=_mixer_config(case),
            ffn=sb.SLinOSSMLPConfig(kind="gelu", expand=4.0, bias=case["bias"]))
        config = sb.SLinOSSStackConfig.uniform(block, n_layers=case["layers"])
        model = SLinOSSLM(case["vocab"], config, device="cuda", dtype=io)
        with torch.no_grad():    # what starts at zero has moved once a model is in training
            for name, p in model.named_parameters():
                if name.endswith(("in_proj.bias", "out_proj.bias", "theta_mod_bias")):
                    p.normal_(0.0, 0.05, generator=gen)
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=gen, device="cuda")
        return {"kind": kind, "trainer": DataParallelTrainer(model, reduce=False), "ids": ids,
                "params": [p.detach() for p in model.parameters()]}
    if kind == "stack_step":
        block = sb.SLinOSSBlockConfig(d_model=case["d_model"], mixer=_mixer_config(case),
                                      ffn=sb.SLinOSSMLPConfig(kind=case["ffn"]))
        stack = sb.SLinOSSStack(sb.SLinOSSStackConfig.uniform(block, n_layers=case["layers"]), device="cuda", dtype=io)
        _init_linear(stack, gen)
        return {"kind": kind, "stack": stack.eval(), "x": rn(case["batch"], case["d_model"]),
                "state": stack.init_decode_state(case["batch"])}
    mixer = sb.SLinOSSMixer(case["d_model"], **_mixer_config(case).build_kwargs(), device="cuda", dtype=io)
    _init_linear(mixer, gen)
    if kind == "mixer_train":
        x = rn(case["batch"], case["seq"], case["d_model"]).requires_grad_(True)
        return {"kind": kind, "mixer": mixer, "x": x, "params": list(mixer.parameters()), "d_out": rn(*x.shape)}
    if kind == "mixer_prefill":
        return {"kind": kind, "mixer": mixer, "x": rn(case["batch"], case["seq"], case["d_model"])}
    x = rn(case["batch"], case["d_model"])
    if kind == "mixer_step":
        return {"kind": kind, "mixer": mixer, "x": x, "state": mixer.init_decode_state(case["batch"])}
    return {"kind": kind, "engine": MixerDecodeEngine(mixer, case["batch"], dtype=io), "x": x}


# ---- one pass -----------------------------------------------------------------------------------------------
def _tensors(state):
    return [state.conv, state.scan.state, state.scan.b_prev, state.scan.u_prev]


def run(state):
    kind = state["kind"]
    if kind == "scan_train":
        ins = state["inputs"]
        args = [ins[k] for k in "UMKBC"]
        carried = {k: ins[k] for k in ("initial_states", "B_prev", "U_prev") if k in ins}
        y = v2x2ssd_cute(*args, chunk_size=CHUNK, **carried)
        return [y, *torch.autograd.grad(y, args + list(carried.values()), state["dY"])]
    if kind == "lm_train":
        return [state["trainer"].step(state["ids"]), *state["params"]]
    if kind == "mixer_train":
        out = state["mixer"](state["x"])
        return [out, *torch.autograd.grad(out, [state["x"], *state["params"]], state["d_out"])]
    if kind == "engine_step":
        engine = state["engine"]
        return [engine.step(state["x"]), *_tensors(engine.state)]
    with torch.no_grad():
        if kind == "scan_prefill":
            ins = state["inputs"]
            carried = {k: ins[k] for k in ("initial_states", "B_prev", "U_prev") if k in ins}
            return list(v2x2ssd(*[ins[k] for k in "UMKBC"], chunk_size=CHUNK, **carried))
        if kind == "scan_decode":
            out = v2x2ssd_decode(*state["token"], state=state["state"], B_prev=state["B_prev"],
                                 U_prev=state["U_prev"], inplace=True)
            return [out[0], out[1]]
        if kind == "mixer_prefill":
            out, carried = state["mixer"](state["x"], return_state=True)
            return [out, *_tensors(carried)]
        if kind == "mixer_step":
            y, carried = state["mixer"].step(state["x"], state["state"], inplace=True)
            return [y, *_tensors(carried)]
        y, carried = state["stack"].step(state["x"], state["state"], inplace=True)
        state["state"] = carried
        return [y] + [t for layer in carried.layers for t in _tensors(layer.mixer)]


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _scan_work(streams, group_streams, seq, N, io, train):
    """Bytes and flops of the scan over ``streams`` = batch * heads sequences: every operand and result once."""
    fwd = streams * seq * (2 * P * io + 24) + group_streams * seq * 2 * 2 * N * io
    bwd = streams * seq * (2 * P * io + 24) + group_streams * seq * 2 * 2 * N * io
    flops = 12 * P * N * streams * seq
    return (fwd + bwd, 3 * flops) if train else (fwd, flops)


def _mixer_work(case, rows, seq):
    """Weights, GEMM flops and the scan of one mixer over ``rows`` tokens; ``seq`` 1: one token over the state."""
    d, N, io = case["d_model"], case["state"], BYTES[case["dtype"]]
    inner = max(1, int(math.floor(case.get("expand", 2.0) * d / P + 0.5))) * P
    heads = inner // P
    groups = case["groups"] or heads
    width = 2 * inner + 3 * heads + 4 * groups * N
    weights = (d * width + inner * d + inner * 6) * io
    flops = 2 * rows * d * (width + inner)
    state = rows // seq * (heads * P * 2 * N * 4 + (inner * 4 + groups * 2 * N) * io)
    return weights, flops + 12 * P * N * heads * rows, state


def work(case):
    kind = case["kind"]
    io = BYTES[case["dtype"]]
    if kind.startswith("scan"):
        streams, group_streams = case["batch"] * case["heads"], case["batch"] * case["groups"]
        nbytes, flops = _scan_work(streams, group_streams, case["seq"], case["state"], io, kind == "scan_train")
        carried = streams * P * 2 * case["state"] * 4
        if kind == "scan_decode" or case["carried"]:
            nbytes += 2 * carried
        elif kind == "scan_prefill":
            nbytes += carried * io // 4
        return {"bytes": nbytes, "flops": flops}
    d, batch = case["d_model"], case["batch"]
    if kind in ("mixer_step", "engine_step"):
        weights, flops, state = _mixer_work(case, batch, 1)
        return {"bytes": weights + 2 * state + 2 * batch * d * io, "flops": flops}
    if kind == "stack_step":
        weights, flops, state = _mixer_work(case, batch, 1)
        hidden = sb.SLinOSSMLPConfig(kind=case["ffn"]).resolve_hidden_dim(d)
        ffn = d * hidden * (3 if case["ffn"] == "swiglu" else 2)
        layer = weights + 2 * state + ffn * io
        return {"bytes": case["layers"] * layer + 2 * batch * d * io,
                "flops": case["layers"] * (flops + 2 * batch * ffn)}
    rows = batch * case["seq"]
    weights, flops, state = _mixer_work(case, rows, case["seq"])
    if kind == "mixer_prefill":
        return {"bytes": weights + 2 * rows * d * io + state * io // 4, "flops": flops}
    if kind == "mixer_train":
        return {"bytes": 2 * weights + 4 * rows * d * io, "flops": 3 * flops}
    ffn = 2 * d * 4 * d
    params = case["layers"] * (weights + ffn * io) + case["vocab"] * d * io
    return {"bytes": 2 * 3 * params + rows * 8,     # parameters and both moments, in and out
            "flops": 3 * (case["layers"] * (flops + 2 * rows * ffn) + 2 * rows * d * case["vocab"])}


def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 2e-5}
    if case["kind"] == "mixer_train":
        return {"rel": 2e-2}    # per-head parameter gradients are sums over every token of terms of both signs
    return {"rel": 1e-2}
