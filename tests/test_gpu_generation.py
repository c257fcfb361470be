"""Decoding through captured steps against steps issued one by one: the same kernels, so the same tokens exactly."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(**kw):
    from kohakuwullm_b200.models import LMBackbone, get_preset
    from kohakuwullm_b200.training.optim.lowbit import cast_parameters_

    torch.manual_seed(0)
    with torch.device("cuda"):
        model = LMBackbone(get_preset(kw.pop("preset", "B200-smoke"), vocab_size=512, **kw))
    cast_parameters_(model, torch.bfloat16)
    model.eval()
    for blk in model.blocks:
        if getattr(blk.attn, "sink", None) is not None:
            torch.nn.init.normal_(blk.attn.sink, std=1.0)
    return model


@pytest.mark.parametrize("kw,rows,prompt,new", [
    ({}, 1, 5, 9), ({}, 3, 250, 14),                                      # the cache crosses a chunk of 256 keys
    (dict(sliding_window=16, global_layer_every=2, attn_sink=True, attn_num_sinks=2), 2, 10, 24),
    (dict(sliding_window=300), 2, 290, 20), (dict(preset="Kohaku-MoE-1B", depth=3), 2, 20, 8),
    (dict(preset="B200-dense-546M", depth=3, mxfp8=True), 3, 20, 8), (dict(preset="Kohaku-MoE-1B", depth=3, mxfp8=True), 2, 20, 8)])
def test_captured_steps_give_the_tokens_of_direct_steps(kw, rows, prompt, new):
    from kohakuwullm_b200.generation.engine import LocalGenerator, StepGraph, capturable
    from kohakuwullm_b200.ops import native

    model = _model(**dict(kw))
    tokens = torch.randint(1, 512, (rows, prompt), device="cuda")
    assert capturable(model, tokens)
    built = []
    original = StepGraph.__init__

    def counting(self, *a):
        original(self, *a)
        built.append(self)

    StepGraph.__init__ = counting
    try:
        for sampling in (dict(temperature=0.0), dict(temperature=0.9, top_p=0.95)):
            fast, direct = LocalGenerator(model, eos_id=511, stop_ids=(600,)), LocalGenerator(model, eos_id=511, stop_ids=(600,))
            got = [fast.generate(tokens, new, **sampling) for _ in range(2)]      # the second call takes the first's memory
            assert len(built) == 2
            hook = model.final_norm.register_forward_hook(lambda *a: None)
            assert not capturable(model, tokens)
            want = [direct.generate(tokens, new, **sampling) for _ in range(2)]
            hook.remove()
            assert len(built) == 2
            built.clear()
            torch.cuda.synchronize()
            native.check_status()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        StepGraph.__init__ = original


def test_models_that_read_back_or_are_altered_are_not_captured():
    from kohakuwullm_b200.generation.engine import capturable

    tokens = torch.ones(1, 4, dtype=torch.long, device="cuda")
    assert not capturable(_model(attn="sdpa"), tokens)
    model = _model()
    assert capturable(model, tokens) and not capturable(model, tokens.cpu())
    model.head.logits = lambda h: h
    assert not capturable(model, tokens)
    assert not capturable(_model().float(), tokens)


def test_modes_see_every_decode_step():
    """A dispatch or function mode (an operation counter) around a call sees all of its steps: none is replayed."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from kohakuwullm_b200.generation.engine import LocalGenerator, capturable

    class Dispatch(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen += 1
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        seen = 0

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen += 1
            return func(*args, **(kwargs or {}))

    model = _model()
    tokens = torch.randint(1, 512, (1, 5), device="cuda")
    gen = LocalGenerator(model, eos_id=511, stop_ids=(600,))
    want = gen.generate(tokens, 24, temperature=0.0)
    for mode in (Dispatch, Function):
        counts = []
        for new in (8, 16, 24):
            with mode() as m:
                assert not capturable(model, tokens)
                got = gen.generate(tokens, new, temperature=0.0)
            counts.append(m.seen)
        assert torch.equal(got, want)
        assert counts[2] - counts[1] == counts[1] - counts[0] > 8 * model.config.depth    # the same for each eight steps
    assert capturable(model, tokens)
