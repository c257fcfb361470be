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


def test_other_threads_draw_random_numbers_while_steps_are_captured():
    """A capture concerns the thread and the stream that it runs on: another thread's draws from the device's default
    generator, allocations and launches go on meanwhile, on as many of torch's streams as there are."""
    import threading

    from kohakuwullm_b200.generation.engine import LocalGenerator
    from kohakuwullm_b200.ops import native

    model = _model()
    tokens = torch.randint(1, 512, (1, 5), device="cuda")
    gen = LocalGenerator(model, eos_id=511, stop_ids=(600,))
    want = gen.generate(tokens, 7, temperature=0.0)
    done, errors = threading.Event(), []

    def draw():
        streams = [torch.cuda.Stream() for _ in range(32)]
        while not done.is_set():
            for stream in streams:
                try:
                    with torch.cuda.stream(stream):
                        assert float(torch.rand(1000, device="cuda").max()) <= 1.0
                    draws.append(1)
                except Exception as err:
                    errors.append(err)
                    return

    draws = []
    other = threading.Thread(target=draw)
    other.start()
    try:
        got = [gen.generate(tokens, 7, temperature=0.0) for _ in range(60)]
    finally:
        done.set()
        other.join()
    torch.cuda.synchronize()
    native.check_status()
    assert not errors, errors[0]
    assert len(draws) > 60 and all(torch.equal(g, want) for g in got)


def test_captures_of_several_calls_take_over_their_memory():
    """Calls after the first reserve no further memory, whatever the rows, and a generator that is dropped leaves none."""
    import gc

    from kohakuwullm_b200.generation.engine import LocalGenerator

    model = _model()
    prompts = [torch.randint(1, 512, (rows, 6), device="cuda") for rows in (4, 1, 3)]
    LocalGenerator(model, eos_id=511, stop_ids=(600,)).generate(prompts[0], 9, temperature=0.0)    # what is made once
    gc.collect()
    torch.cuda.empty_cache()
    start = torch.cuda.memory_allocated()
    gen = LocalGenerator(model, eos_id=511, stop_ids=(600,))
    first = [gen.generate(p, 9, temperature=0.0) for p in prompts]
    reserved = torch.cuda.memory_reserved()
    for _ in range(5):
        assert all(torch.equal(gen.generate(p, 9, temperature=0.0), f) for p, f in zip(prompts, first))
    assert torch.cuda.memory_reserved() == reserved
    del gen, first
    gc.collect()
    assert torch.cuda.memory_allocated() == start
    torch.cuda.empty_cache()
    assert torch.cuda.memory_reserved() < reserved


def test_a_preview_leaves_no_memory_behind():
    """The sampler of the in-training previews lives as long as the trainer and keeps no capture's memory from training."""
    import gc

    from kohakuwullm_b200.training.loop.sampling import PreviewSampler

    class Tok:
        bos_token_id = None
        encode = staticmethod(lambda text: [ord(c) for c in text])
        decode = staticmethod(lambda ids: " ".join(map(str, ids)))

    model = _model()
    prompt = torch.randint(1, 512, (2, 6), device="cuda")
    sampler = PreviewSampler(eos_id=511)
    for call in (lambda: sampler.generate(model, prompt, 9, temperature=0.0),
                 lambda: sampler.texts(model, Tok, ["ab", "xyz"], 9, count=2, temperature=0.0)):
        call()                                       # what is made once
        gc.collect()
        torch.cuda.empty_cache()
        start = torch.cuda.memory_reserved()
        call()
        gc.collect()
        torch.cuda.empty_cache()
        assert torch.cuda.memory_reserved() == start and not sampler._pools
