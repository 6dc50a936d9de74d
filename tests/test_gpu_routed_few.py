"""Routed experts of few pairs: the products that stream the chosen experts' weights."""

import os

import pytest
import torch

from test_gpu_routed_wide import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,ff", [(72, 16), (264, 144), (1032, 272), (2080, 48)])
@pytest.mark.parametrize("tokens", [1, 8, 9, 20, 21])
@pytest.mark.parametrize("weight_inputs", [False, True])
def test_few_pairs(tokens, hidden, ff, weight_inputs):
    """An expert that every token chooses (units of eight pairs, one more, two and a half), one that none does; k that ends
    inside a block of 32, with fewer blocks than warps and with several steps a warp; weight rows that end inside a unit.  A
    token alone gives the same bits.  The activation is rounded to bfloat16 once, the sums are float32: 2^-7 of the largest."""
    check_few(tokens, hidden, ff, weight_inputs)


@pytest.mark.parametrize("hidden,ff", [(72, 16), (264, 144)])
@pytest.mark.parametrize("tokens", [1, 2, 21])
@pytest.mark.parametrize("tcgen05", ["0", "1"])
def test_few_pairs_on_the_grouped_products(monkeypatch, tokens, hidden, ff, tcgen05):
    """The same with the kernel for few pairs off: a plan for a single token, too, alone and among others (as above)."""
    monkeypatch.setenv("CIE_MOE_FEW", "0")
    monkeypatch.setenv("CIE_MOE_TCGEN05", tcgen05)
    check_few(tokens, hidden, ff, False)


def check_few(tokens, hidden, ff, weight_inputs):
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", "bfloat16")
    rt.ops._load_moe()
    experts, top = 6, 3
    x = rand(tokens, hidden, seed=1).bfloat16()
    router, bias = rand(experts, hidden, seed=2, scale=0.3), torch.tensor([0.0, 90.0, -90.0, 0.5, 0.0, -1.0])
    gate, up = (rand(experts, ff, hidden, seed=s, scale=hidden ** -0.5).bfloat16() for s in (3, 4))
    down = rand(experts, hidden, ff, seed=5, scale=ff ** -0.5).bfloat16()
    assert rt.ops.moe_interleaves(hidden, ff) and (tokens * top <= rt.ops.moe_few_pairs or os.environ.get("CIE_MOE_FEW") == "0")
    both = rt.ops.interleave_gate_up(gate.cuda(), up.cuda())

    def run(rows):
        out = torch.full((rows.shape[0] + 1, hidden), 7.0).cuda()
        rt.ops.routed_experts(rows.cuda(), router.cuda(), None, both, None, down.cuda(), top, False, out[:-1], rt.workspace,
                              router_bias=bias.cuda(), chosen_softmax=True, weight_inputs=weight_inputs)
        rt.ops.check_errors()
        assert float((out[-1] - 7.0).abs().max()) == 0
        return out[:-1].cpu()

    out = run(x)
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
    assert float((out.double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
    for t in range(tokens):
        assert torch.equal(run(x[t:t + 1])[0], out[t])


@pytest.mark.parametrize("hidden,ff,most", [(2048, 1376, 1.0e-7), (4096, 2048, 1.1e-7)])
def test_rows_of_few_pairs_are_as_far_from_64_bits_as_float32_sums(hidden, ff, most):
    """The down product's float32 rows against 64 bits, from the activations as they were rounded, over their norm: 8.6e-8 and 9.2e-8
    (8.4e-8 and 9.5e-8 as one FMA after the other; sums that the tensor core cuts every 16 columns have 1.31e-7 and 1.75e-7)."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", "bfloat16")
    rt.ops._load_moe()
    tokens, experts, top = 8, 16, 4
    generator = torch.Generator(device="cuda").manual_seed(1)
    normal = lambda *shape: torch.empty(*shape, device="cuda").normal_(0, 0.02, generator=generator)  # noqa: E731
    x, router = (50 * normal(tokens, hidden)).bfloat16(), normal(experts, hidden)
    both = rt.ops.interleave_gate_up(normal(experts, ff, hidden).bfloat16(), normal(experts, ff, hidden).bfloat16())
    down = normal(experts, hidden, ff).bfloat16()
    out = torch.empty(tokens, hidden, device="cuda")
    rt.ops.routed_experts(x, router, None, both, None, down, top, False, out, rt.workspace, chosen_softmax=True)
    rt.ops.check_errors()
    assert tokens * top <= rt.ops.moe_few_pairs
    ids = rt.workspace.get("moe.ids", tokens, top, torch.int32).view(-1).long()
    act = rt.workspace.get("moe.act", tokens, top * ff, rt.dtype).view(-1, ff)
    rows = rt.workspace.get("moe.rows", tokens, top * hidden, torch.float32).view(-1, hidden)
    want = torch.einsum("pf,phf->ph", act.double(), down[ids].double())
    error = float((rows.double() - want).norm() / want.norm())
    print(f"{hidden} x {ff}: {error:.3e}")
    assert error <= most
