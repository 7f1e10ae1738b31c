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
