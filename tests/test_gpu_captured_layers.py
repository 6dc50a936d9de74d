"""Layers that keep a state, decoding from a captured graph: a replay is a function of its input and the state it finds."""

import importlib.util
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

spec = importlib.util.spec_from_file_location("perf_cases", Path(__file__).resolve().parent.parent / "perf" / "cases.py")
cases = importlib.util.module_from_spec(spec)
spec.loader.exec_module(cases)


def captured(case, seed):
    """The layer's call on single tokens in a graph that begins by putting the state back; everything that it reads is kept."""
    from cloud_inference_from_scratch_b200 import models, parts  # noqa: F401
    from cloud_inference_from_scratch_b200.engine.core import build_core
    from cloud_inference_from_scratch_b200.engine.step import StepEntry

    batch = cases.requests(case)
    core = build_core(None, dtype="bfloat16", page_size=16, num_pages=600, max_requests=len(batch), max_model_len=4096,
                      max_tokens_per_step=0, random_config=cases._configuration(case), seed=1, random_device="cuda")
    mixer = core.model.layers[0].mixer
    mixer.bind(cases._weights(case, seed), core.runtime)
    for i in range(len(batch)):
        core.step.admit(i)
    core.cache.ensure_capacity_batch({i: (0, before) for i, (_, before) in enumerate(batch)})
    core.cache.commit_lengths({i: before for i, (_, before) in enumerate(batch)})
    host, _, _ = core.step.prepare([StepEntry(i, [0], want=()) for i in range(len(batch))])
    ctx = core.step.upload(host)
    binding = ctx.bindings[0]
    start = torch.zeros_like(binding.state)
    for i, (_, before) in enumerate(batch):
        start[core.cache.slot(i)] = cases._state_of(case, seed, i, before).view(start[0].shape)
    x = cases._inputs(case, seed, case["width"])
    outputs = []

    def call():
        binding.state.copy_(start)
        outputs[:] = [mixer.forward(x, ctx, binding), binding.state]

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    return core, ctx, x, start, graph, outputs


@pytest.mark.parametrize("decode,context", [(1, 30), (9, 500)])
@pytest.mark.parametrize("width", [2048, 4096])
@pytest.mark.parametrize("kind", ["delta", "gated_delta", "gla"])
def test_replays_of_a_decode_layer_give_the_same_bits(kind, width, decode, context):
    """Three replays, another layer of the kind built and run between them; the outputs and the state after the token
    against the same in 64 bits.  bfloat16 rounds the inputs of the products: a hundredth, as for the layer's prompts."""
    case = dict(kind=kind, width=width, style="", dtype="bfloat16", decode=decode, portions=0, tokens=0, context=context)
    held = captured(case, 3)
    graph, outputs = held[4:]
    seen = []
    for other_seed in (None, 4, 5):
        if other_seed is not None:
            other = captured(case, other_seed)
            other[4].replay()
        graph.replay()
        torch.cuda.synchronize()
        held[0].runtime.ops.check_errors()
        seen.append([t.clone() for t in outputs])
    for again in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(again, seen[0]))
    for got, want in zip(seen[0], cases.exact(case, 3)):
        off = (got.double().reshape(-1) - want.reshape(-1)).norm() / want.norm()
        assert float(off) < 0.01
