"""What a native token plan keeps alive and what it notices, without a GPU: plans are made on CPU modules and checked, not run."""

import gc
import weakref

import pytest
import torch

import slinoss_b200 as sb


def _mixer():
    return sb.SLinOSSMixer(64, d_state=64, d_head=64, dtype=torch.bfloat16)


def _block(ffn=True):
    return sb.SLinOSSBlock(sb.SLinOSSBlockConfig(
        d_model=64, mixer=sb.SLinOSSMixerConfig(d_state=64, d_head=64),
        ffn=sb.SLinOSSMLPConfig(kind="gelu", multiple_of=8) if ffn else None), dtype=torch.bfloat16)


def _planned(module):
    """The module with its plan, and those of its parts, where ``step`` keeps them."""
    for m in (module, getattr(module, "mixer", None)):
        if m is not None:
            m.__dict__["_token_plan"] = m._make_token_plan()
            assert m.__dict__["_token_plan"].valid(m.__dict__)
    return module


MAKE = [_mixer, _block, lambda: _block(ffn=False)]


@pytest.mark.parametrize("make", MAKE)
def test_a_plan_does_not_keep_its_module_alive(make):
    """Parameters go with the module at once, as without a plan, and with the next collection where the program has put the
    module on a cycle of its own."""
    for cycle in (False, True):
        module = _planned(make())
        if cycle:
            module.__dict__["neighbour"] = [module]
            getattr(module, "mixer", module).__dict__["owner"] = [module]
        alive = [weakref.ref(p) for p in module.parameters()]
        storage = [weakref.ref(p.untyped_storage()) for p in module.parameters()]
        gc.collect()
        gc.disable()
        try:
            del module
            if cycle:
                gc.collect()
            assert not any(r() is not None for r in alive + storage)
        finally:
            gc.enable()


def _replace_step(module):
    module.__dict__["step"] = lambda *a, **k: None


@pytest.mark.parametrize("part, change, undo", [
    ("mixer.out_norm", lambda m: setattr(m, "eps", 0.5), None),
    ("mixer_norm", lambda m: setattr(m, "eps", 0.5), None),
    ("ffn_norm", lambda m: setattr(m, "eps", 0.5), None),
    ("mixer", _replace_step, "step"),
    ("mixer.out_proj", lambda m: m.__dict__.update(forward=lambda x: x), "forward"),
    ("ffn", lambda m: m.__dict__.update(forward=lambda x: x), "forward"),
    ("ffn.in_proj", lambda m: m.__dict__.update(forward=lambda x: x), "forward"),
    ("mixer_norm", lambda m: m.__dict__.update(forward=lambda x: x), "forward"),
    ("ffn", lambda m: m.register_forward_hook(lambda *a: None), None),
])
def test_a_plan_notices_values_and_methods_that_it_relies_on(part, change, undo):
    block = _planned(_block())
    plan, target = block.__dict__["_token_plan"], block.get_submodule(part)
    change(target)
    assert not plan.valid(block.__dict__)
    if part == "mixer.out_norm":
        assert not block.mixer.__dict__["_token_plan"].valid(block.mixer.__dict__)
    if undo is not None:
        assert block._make_token_plan() is None    # the composed path, as long as the replacement is there
        del target.__dict__[undo]
        assert plan.valid(block.__dict__)


def test_a_hook_on_every_module_ends_a_plan():
    block = _planned(_block())
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert not block.__dict__["_token_plan"].valid(block.__dict__) and block._make_token_plan() is None
    finally:
        handle.remove()
    assert block.__dict__["_token_plan"].valid(block.__dict__)


def test_an_epsilon_that_follows_the_type_makes_no_plan():
    block = _block()
    block.mixer.out_norm.eps = None
    assert block._make_token_plan() is None and block.mixer._make_token_plan() is None


def test_a_step_replaced_on_an_instance_is_called_by_the_stack():
    cfg = sb.SLinOSSStackConfig.uniform(_block().config, n_layers=2)
    stack = sb.SLinOSSStack(cfg, dtype=torch.bfloat16).eval()
    stack.blocks[1].__dict__["step"] = lambda x, state=None, **k: (x + 1, state)
    x = torch.randn(3, 64, dtype=torch.bfloat16)
    stack.blocks[0].__dict__["step"] = lambda x, state=None, **k: (x * 2, state)
    with torch.no_grad():
        y, _ = stack.step(x, stack.init_decode_state(3))
    assert torch.equal(y, stack.final_norm(x * 2 + 1))
