"""Which passes may read the cache ahead of a kernel's wait: those behind a copy of their own batch, and no others."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from research_2_b200.engine import step
from research_2_b200.engine.batch import batch_for


class Event:
    def __init__(self, name):
        self.name, self.recorded = name, 0

    def record(self):
        self.recorded += 1


class Order:
    begin = end = staticmethod(lambda *a: None)


def one_row_batch():
    batch = batch_for((4,), 1, 1, 1)
    batch.set_entries([0], [0], [[3]])
    batch.set_logit_rows([0])
    batch.trusted = True
    return batch


def context(batch):
    return step.StepContext(batch, torch.from_numpy(batch.buf.copy()))


def test_a_context_that_was_uploaded_earlier_is_not_settled():
    assert context(one_row_batch()).cache_settled is False


@pytest.mark.parametrize("entry", ["__call__", "step_and_sample"])
def test_the_step_function_settles_the_pass_behind_its_own_copy(entry, monkeypatch):
    monkeypatch.setattr(step.torch.cuda, "device", lambda d: torch.no_grad())
    monkeypatch.setattr(step.torch.cuda, "is_current_stream_capturing", lambda: False)
    fn, seen = step.StepFunction.__new__(step.StepFunction), []
    fn.capture, fn._graphs, fn.device, fn._device_index, fn._pass_done = False, {}, "cpu", 0, Event("pass")
    fn.order = Order()
    fn.upload, fn.sample = context, lambda logits, ctx: logits
    fn.forward = lambda ctx: seen.append(ctx.cache_settled)
    batch = one_row_batch()
    getattr(fn, entry)(batch)
    assert seen == [True]
    assert fn.upload(batch).cache_settled is False   # (what a caller uploads)


def test_a_pass_on_another_stream_waits_for_the_one_before(monkeypatch):
    """Whichever graph the one before was, and where it was none."""
    current, waits = [7], []

    class Stream:
        wait_event = staticmethod(lambda event: waits.append((current[0], event.name)))

    monkeypatch.setattr(step.torch._C, "_cuda_getCurrentRawStream", lambda i: current[0])
    monkeypatch.setattr(step.torch.cuda, "current_stream", lambda d=None: Stream)
    monkeypatch.setattr(step.torch.cuda, "device", lambda d: torch.no_grad())
    monkeypatch.setattr(step.torch.cuda, "is_current_stream_capturing", lambda: False)
    fn = step.StepFunction.__new__(step.StepFunction)
    fn.capture, fn._graphs, fn.device, fn._device_index, fn._pass_done = False, {}, "cpu", 0, Event("eager")
    fn.order = step.PassOrder("cpu", 0)
    fn.upload, fn.forward = context, lambda ctx: None

    def graph(name):
        g = step.StepGraph.__new__(step.StepGraph)
        g.order, g.turn, g.kernels, g.done = fn.order, 0, 0, None
        g.hosts = [one_row_batch(), one_row_batch()]
        for i, host in enumerate(g.hosts):
            host.copy_done = Event(f"{name} {i}")
            host.copy_done.synchronize = lambda: None
        g.graph = type("Graph", (), {"replay": staticmethod(lambda: None)})
        return g

    prompt, decode = graph("prompt"), graph("decode")
    for launch, stream in [(prompt, 7), (decode, 7), (prompt, 7), (decode, 9), (decode, 9), (prompt, 7), (None, 9), (None, 9), (decode, 7), (None, 7)]:
        current[0] = stream
        if launch is None:
            fn(one_row_batch())
        else:
            launch.replay(launch.host)
    assert waits == [(9, "prompt 1"), (7, "decode 0"), (9, "prompt 0"), (7, "eager")]


def test_a_pass_in_a_callers_own_graph_waits_for_nothing_outside_it(monkeypatch):
    """(An event recorded outside a capture ends the capture with an error.)"""
    calls = []

    class Recorder:
        begin = staticmethod(lambda: calls.append("begin"))
        end = staticmethod(lambda event: calls.append("end"))

    monkeypatch.setattr(step.torch.cuda, "device", lambda d: torch.no_grad())
    fn = step.StepFunction.__new__(step.StepFunction)
    fn.capture, fn._graphs, fn.device, fn._device_index, fn._pass_done = False, {}, "cpu", 0, Event("eager")
    fn.order, fn.upload, fn.forward = Recorder(), context, lambda ctx: None
    for capturing in (True, False):
        monkeypatch.setattr(step.torch.cuda, "is_current_stream_capturing", lambda: capturing)
        fn(one_row_batch())
        assert calls == ([] if capturing else ["begin", "end"])


def test_a_graph_made_on_another_stream_waits_for_the_pass_before(monkeypatch):
    """Its warm-up passes write the same workspaces and pad pages."""
    calls = []

    class Recorder:
        begin = staticmethod(lambda: calls.append("begin"))

    monkeypatch.setattr(step.torch.cuda, "device", lambda d: torch.no_grad())
    monkeypatch.setattr(step, "StepGraph", lambda *a: calls.append("warm-up"))
    fn = step.StepFunction.__new__(step.StepFunction)
    fn._graphs, fn.device, fn.order = {}, "cpu", Recorder()
    fn._graph(4, 4)
    assert calls == ["begin", "warm-up"]


def test_the_embedding_is_launched_in_plain_order(monkeypatch):
    from research_2_b200.parts import Runtime, embedding

    orders = []
    monkeypatch.setattr(embedding.ops, "embed", lambda *a, plain_order=False, **k: orders.append(plain_order))
    embedding.TokenEmbedding(torch.zeros(10, 4), Runtime(torch.device("cpu"), torch.float32)).forward(context(one_row_batch()))
    assert orders == [True]


@pytest.mark.gpu
def test_two_contexts_uploaded_before_either_pass():
    """The second pass reads the key and value that the first one writes; neither copy lies between them."""
    from research_2_b200.cache.manager import CacheManager
    from research_2_b200.parts import PartSpec, Runtime, build_part

    dev, heads, hd, width, steps = torch.device("cuda:0"), 4, 64, 256, 12
    gen = torch.Generator().manual_seed(0)
    tensors = {"w": torch.randn(width, 3 * heads * hd, generator=gen) * width ** -0.5, "b": torch.randn(3 * heads * hd, generator=gen) * 0.1,
               "o": torch.randn(heads * hd, width, generator=gen) * width ** -0.5, "ob": torch.zeros(width)}
    part = build_part("mixer", PartSpec("attention", {"n_heads": heads, "n_kv_heads": heads, "head_dim": hd, "scale": hd ** -0.5, "window": 0},
                                        {"w_qkv": "w", "b_qkv": "b", "w_out": "o", "b_out": "ob"}), tensors, Runtime(dev, torch.bfloat16))

    class Shell:
        rt, cache_members, state_members, max_seq_len, vocab_size, blocks = Runtime(dev, torch.bfloat16), [part.cache_spec], [], 128, 10, []

    def logits(ahead: bool):
        fn = step.StepFunction(Shell, 16, 16, 1)
        cache = CacheManager(fn.cache_groups(), 1, 128)
        fn.arena.fill_(64.0)   # (a row that is read before it is written shows)
        cache.open(0)
        cache.reserve(0, 0, steps)
        contexts = []
        for i in range(steps):
            batch = fn.new_batch(1, 1, 1)
            batch.set_entries([0], [i], [[0]])
            cache.fill(batch)
            batch.set_logit_rows([0])
            contexts.append(fn.upload(batch))
        h = torch.randn(steps, width, generator=torch.Generator().manual_seed(1)).to(dev)
        rows, residual = h.bfloat16(), h.clone()
        torch.cuda.synchronize()   # from here on nothing is launched but the passes' own kernels
        out = []
        for i, ctx in enumerate(contexts):
            out.append(part.forward(rows[i: i + 1], residual[i: i + 1], ctx, fn.arena.members[0]))
            if not ahead:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return torch.cat(out)

    want = logits(False)
    assert torch.isfinite(want).all() and np.isfinite(float(want.abs().max()))
    assert torch.equal(logits(True), want)


@pytest.mark.gpu
def test_a_pass_in_a_callers_own_graph(tmp_path):
    import research_2_b200 as r2
    from tests.helpers import TINY_B, make_model_dir, random_tokens

    folder = make_model_dir(tmp_path / "tiny", TINY_B, std=0.2)
    with r2.run(folder, dtype="bfloat16", block_size=16, max_requests=1, max_batch_tokens=64, capture=False) as engine:
        engine.submit(random_tokens(5, 40, 512), 4)
        batch = engine.build_batch(engine.plan())
        want = engine.step_fn(batch).clone()   # on the current stream; a capture has one of its own
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = engine.step_fn(batch)
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
