"""Steps that run as CUDA graphs are launched while the one before still runs: their batches come from two host buffers in turn."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import TINY_B, make_model_dir, random_tokens

pytestmark = pytest.mark.gpu


def replayed(folder, capture: bool, dtype: str):
    """Logits of every step of three requests whose tokens are given, no step waited for; and of the last batch run once more."""
    import research_2_b200 as r2

    prompts = [random_tokens(40 + i, n, 512) for i, n in enumerate((70, 9, 33))]
    replies = np.random.default_rng(5).integers(0, 512, (3, 20), dtype=np.int32)
    out = []
    with r2.run(folder, dtype=dtype, block_size=16, max_requests=3, max_batch_tokens=64, capture=capture) as engine:
        engine.step_fn.capture_after = 0
        index = {engine.submit(p, 20): i for i, p in enumerate(prompts)}
        while (plan := engine.plan()) is not None:
            batch = engine.build_batch(plan)
            out.append(engine.step_fn(batch).clone())
            tokens = np.zeros(plan.n_entries, dtype=np.int32)
            for e in range(plan.n_entries):
                i = index[int(plan.req[e])]
                if plan.emits[e]:
                    tokens[e] = replies[i][int(plan.start[e] + plan.rows[e]) - len(prompts[i])]
            engine.commit(tokens)
        if capture:
            assert engine.step_fn._graphs
        out.append(engine.step_fn(batch).clone())   # the same batch again: by now it is the other buffer's turn
        other = torch.cuda.Stream()
        other.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(other):               # and on another stream, while the one before may still run
            out.append(engine.step_fn(batch).clone())
        torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_graph_steps_launched_ahead_give_the_logits_of_eager_ones(tmp_path, dtype):
    folder = make_model_dir(tmp_path / "tiny", TINY_B, std=0.2)
    eager, graphs = replayed(folder, False, dtype), replayed(folder, True, dtype)
    assert len(eager) == len(graphs) > 20
    for a, b in zip(eager, graphs):
        if dtype == "float32":
            assert torch.equal(a, b)
        else:   # (padded steps may choose other kernels: two roundings of the logits' size apart)
            torch.testing.assert_close(a, b, atol=2.0 ** -5 * float(a.abs().max()), rtol=0.0)
    assert torch.equal(graphs[-1], graphs[-2])


@pytest.mark.parametrize("capture", [False, True])
def test_steps_on_two_streams_in_turn(tmp_path, capture):
    """Every pass, whichever graph or single launches it takes, waits for the one before, whose caches and buffers it uses: nobody else orders the streams."""
    import research_2_b200 as r2

    folder = make_model_dir(tmp_path / "tiny", TINY_B, std=0.2)
    prompts = [random_tokens(60 + i, n, 512) for i, n in enumerate((70, 9, 33))]

    def logits(streams):
        out = []
        with r2.run(folder, dtype="bfloat16", block_size=16, max_requests=3, max_batch_tokens=64, capture=capture) as engine:
            engine.step_fn.capture_after = 0
            for p in prompts:
                engine.submit(p, 20)
            torch.cuda.synchronize()
            while (plan := engine.plan()) is not None:
                batch = engine.build_batch(plan)
                with torch.cuda.stream(streams[len(out) % len(streams)]):
                    out.append(engine.step_fn(batch).clone())
                engine.commit(np.full(plan.n_entries, len(out) % 512, dtype=np.int32))
            torch.cuda.synchronize()
        return out

    one, two = logits([torch.cuda.current_stream()]), logits([torch.cuda.Stream(), torch.cuda.Stream()])
    assert len(one) == len(two) > 20
    assert all(torch.equal(a, b) for a, b in zip(one, two))
