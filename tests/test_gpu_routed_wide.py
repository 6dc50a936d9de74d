"""Routed experts of many pairs: the router that shares its matrix among tokens, and the grouped products in tiles of
128 columns and of 256."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(*shape, seed, scale=1.0):
    generator = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=generator) * scale


@pytest.mark.parametrize("columns", ["128", "256"])
@pytest.mark.parametrize("tokens", [342, 1185])          # one token more than whole blocks of four in the router
@pytest.mark.parametrize("hidden,ff", [(72, 16), (256, 128), (264, 144), (512, 272)])
@pytest.mark.parametrize("weight_inputs", [False, True])
def test_many_pairs(monkeypatch, tokens, hidden, ff, weight_inputs, columns):
    """An expert that every token chooses, one that none does, uneven others; columns that end inside a tile, at its edge
    and one channel block behind it; K that ends inside a step.  The choice is the 32-bit logits' (no two are near a tie
    here); the activation is rounded to bfloat16 once, the sums are float32: 2^-7 of the largest value."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    monkeypatch.setenv("CIE_MOE_TILE_COLUMNS", columns)
    rt = Runtime("cuda:0", "bfloat16")
    experts, top = 6, 3
    x = rand(tokens, hidden, seed=1).bfloat16()
    router, bias = rand(experts, hidden, seed=2, scale=0.3), torch.tensor([0.0, 60.0, -60.0, 0.5, 0.0, -1.0])
    gate, up = (rand(experts, ff, hidden, seed=s, scale=hidden ** -0.5).bfloat16() for s in (3, 4))
    down = rand(experts, hidden, ff, seed=5, scale=ff ** -0.5).bfloat16()
    assert rt.ops.moe_interleaves(hidden, ff)
    both = rt.ops.interleave_gate_up(gate.cuda(), up.cuda())
    out = torch.full((tokens + 1, hidden), 7.0).cuda()
    rt.ops.routed_experts(x.cuda(), router.cuda(), None, both, None, down.cuda(), top, False, out[:tokens], rt.workspace,
                          router_bias=bias.cuda(), chosen_softmax=True, weight_inputs=weight_inputs)
    rt.ops.check_errors()
    logits = x.double() @ router.double().T + bias.double()
    best, chosen = torch.topk(logits, top, dim=1)
    assert bool((chosen == 1).any(1).all()) and not bool((chosen == 2).any())
    share = torch.softmax(best, dim=1)
    want = torch.zeros(tokens, hidden, dtype=torch.float64)
    for e in range(experts):
        token, place = torch.nonzero(chosen == e, as_tuple=True)
        rows, weight = x[token].double(), share[token, place].unsqueeze(1)
        if weight_inputs:
            rows = rows * weight
        g = rows @ gate[e].double().T
        y = (g * torch.sigmoid(g) * (rows @ up[e].double().T)) @ down[e].double().T
        want[token] += y if weight_inputs else weight * y
    assert float((out[:tokens].double().cpu() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
    assert float((out[tokens] - 7.0).abs().max()) == 0
