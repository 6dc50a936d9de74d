"""Routed experts of many pairs: the router that shares its matrix among tokens, and the grouped products in tiles of 128
weight rows by up to 256 tokens of an expert."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(*shape, seed, scale=1.0):
    generator = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=generator) * scale


# pairs of the expert that every token chooses: one short of a tile, a whole one, one more than one and two whole ones, some that
# divide into even tiles, and one token more than whole blocks of four in the router
@pytest.mark.parametrize("tokens", [255, 256, 257, 342, 513, 1185])
@pytest.mark.parametrize("hidden,ff", [(72, 16), (256, 128), (264, 144), (512, 272)])
@pytest.mark.parametrize("weight_inputs", [False, True])
def test_many_pairs(tokens, hidden, ff, weight_inputs):
    """An expert that every token chooses, one that none does, uneven others; weight rows that end inside a tile of 128, at its
    edge and one channel block behind it; K that ends inside a step.  The choice is the 32-bit logits' (no two are near a tie
    here); the activation is rounded to bfloat16 once, the sums are float32: 2^-7 of the largest value."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

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


@pytest.mark.parametrize("activation", [None, (130.0, 1.5, 1.0)])
def test_gates_of_any_size(activation):
    """The activation of the grouped products over gates from -136 to 136, most of all where the exponential is near the largest
    float32 (1 + e^88 and the like), and gates that are infinite.  Float32 and rounded to bfloat16 once: 2^-8 and a little of
    the value (an exponent of 136 is off by half a unit of its last place, 2^-18); where the exponential
    is beyond the largest float32, 2^128, the quotient may be zero."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", "bfloat16")
    rt.ops._load_moe()
    tokens, hidden, ff, experts = 130, 64, 272, 2
    limit, slope, shift = activation or (float("inf"), 1.0, 0.0)
    x = torch.zeros(tokens, hidden)
    x[:, 0] = 1 + (torch.arange(tokens) % 64) / 128          # a token's gates are its one element times the weights
    x[-1, 0] = 4.0
    gates = torch.linspace(-90, 90, ff).bfloat16()
    gates[7], gates[200] = 3e38, -3e38          # infinite for the last token
    gate, up = torch.zeros(experts, ff, hidden), torch.zeros(experts, ff, hidden)
    gate[:, :, 0], up[:, :, 1] = gates.float(), 2.0 ** 60
    x[:, 1] = 1.0
    x, down = x.bfloat16(), torch.zeros(experts, hidden, ff).bfloat16().cuda()
    router = torch.zeros(experts, hidden)
    router[0, 0], router[1, 0] = 1.0, -1.0          # all tokens to expert 0: places are in some order of the tokens
    both = rt.ops.interleave_gate_up(gate.bfloat16().cuda(), up.bfloat16().cuda())
    out = torch.empty(tokens, hidden).cuda()
    rt.ops.routed_experts(x.cuda(), router.cuda(), None, both, None, down, 1, False, out, rt.workspace, chosen_softmax=True,
                          activation=activation)
    rt.ops.check_errors()
    assert tokens > rt.ops.moe_few_pairs
    places = rt.workspace.get("moe.places", tokens, 1, torch.int32).view(-1).long().cpu()
    got = rt.workspace.get("moe.act", tokens, ff, torch.bfloat16).cpu()
    got[places] = got.clone()
    g = (x[:, :1].float() * gates.float()).double().clamp(max=limit)
    u = min(2.0 ** 60, limit) + shift
    want = g / (1 + torch.exp(-slope * g)) * u
    whole = torch.isfinite(g) & (want.abs() < 3e38)
    error = (got.double() - want).abs()[whole]
    assert bool((error <= want.abs()[whole] * (2.0 ** -8 + 2.0 ** -16) + (2.0 ** -127 * g.abs() * u)[whole]).all())
    large = whole & (-slope * g > 87.4) & (-slope * g < 88.7)          # the quotient is a normal float32, about 1e-36
    assert int(large.sum()) > 50 and bool((got[large] != 0).all())
    assert bool(((got[-1, 7] == float("inf")) if activation is None else torch.isfinite(got[-1, 7])).all())
    assert bool(got[-1, 200].isnan())          # -inf / (1 + inf)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("hidden", [70, 72, 1032])          # single elements, pieces of four, several loads a lane
@pytest.mark.parametrize("kind", ["softmax", "sigmoid", "grouped"])
def test_a_router_block_of_four_tokens_adds_like_one_of_a_single_token(kind, hidden, dtype):
    """1,185 tokens at once (four a block, one alone in the last) and 500 at a time (one a block): the same choices and the
    same bits of their weights."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", dtype)
    rt.ops._load_moe()
    tokens, experts, top = 1185, 12, 3
    x = rand(tokens, hidden, seed=1).to(rt.dtype).cuda()
    router, bias, correction = rand(experts, hidden, seed=2).cuda(), rand(experts, seed=3).cuda(), rand(experts, seed=4).cuda()
    pointer = lambda t, wanted=True: t.data_ptr() if wanted else None  # noqa: E731

    def route(rows):
        ids = torch.empty(rows.shape[0], top, dtype=torch.int32).cuda()
        weights = torch.empty(rows.shape[0], top).cuda()
        rt.ops._moe_route(rows.data_ptr(), router.data_ptr(), pointer(correction, kind != "softmax"), ids.data_ptr(),
                          weights.data_ptr(), None, None, None, None, None, None, rows.shape[0], hidden, experts, top, 1,
                          pointer(bias, kind == "softmax"), int(kind == "softmax"), int(kind == "sigmoid"),
                          3 if kind == "grouped" else 1, 2 if kind == "grouped" else 1, 1e-20, rt.ops._code_of(x), rt.ops.stream)
        return ids, weights

    together = route(x)
    apart = [route(x[first:first + 500]) for first in range(0, tokens, 500)]
    for whole, pieces in zip(together, zip(*apart)):
        assert torch.equal(whole, torch.cat(pieces))


@pytest.mark.parametrize("hidden,weighted", [(72, True), (72, False), (4096, True)])
def test_the_sum_of_the_experts_rows_in_pieces_and_element_by_element(hidden, weighted):
    """Rows that begin on 16 bytes and rows that do not: the same additions in the same order."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    ops = Runtime("cuda:0", "bfloat16").ops
    ops._load_moe()
    tokens, top = 37, 5
    values, weights = rand(tokens * top * hidden, seed=1).cuda(), rand(tokens, top, seed=2).cuda()
    results = []
    for shift in (0, 1):
        rows = torch.zeros(values.numel() + 4).cuda()
        rows[shift:shift + values.numel()] = values
        out = torch.full((tokens + 1, hidden), 7.0).cuda()
        ops._moe_combine(rows[shift:].data_ptr(), weights.data_ptr() if weighted else None, out.data_ptr(), tokens, hidden, top,
                         ops._code_of(out), ops.stream)
        results.append(out)
    assert torch.equal(*results) and float((results[0][tokens] - 7.0).abs().max()) == 0


@pytest.mark.parametrize("tokens", [37, 1185])          # a token a block, and four
@pytest.mark.parametrize("kind", ["softmax", "scores", "sigmoid", "grouped"])
def test_tokens_whose_logits_are_nan_or_infinite(kind, tokens):
    """They get experts that there are, each once, and nobody beside them notices."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", "bfloat16")
    rt.ops._load_moe()
    hidden, experts, top = 64, 12, 3
    x = rand(tokens, hidden, seed=1).bfloat16()
    router, correction = rand(experts, hidden, seed=2).cuda(), rand(experts, seed=4).cuda()
    results = []
    for broken in (False, True):
        rows = x.clone()
        if broken:
            rows[1::8, 5], rows[2::8], rows[7::8, 0] = float("nan"), float("inf"), -float("inf")
        rows = rows.cuda()
        ids = torch.empty(tokens, top, dtype=torch.int32).cuda()
        weights = torch.empty(tokens, top).cuda()
        rt.ops._moe_route(rows.data_ptr(), router.data_ptr(), correction.data_ptr() if kind == "grouped" else None,
                          ids.data_ptr(), weights.data_ptr(), None, None, None, None, None, None, tokens, hidden, experts, top, 1,
                          None, int(kind == "softmax"), int(kind in ("sigmoid", "grouped")), 3 if kind == "grouped" else 1,
                          2 if kind == "grouped" else 1, 1e-20, rt.ops._code_of(rows), rt.ops.stream)
        results.append((ids.cpu(), weights.cpu()))
    whole = [t for t in range(tokens) if t % 8 not in (1, 2, 7)]
    for plain, beside in zip(*results):
        assert torch.equal(plain[whole], beside[whole])
    ids = results[1][0].long()
    assert int(ids.min()) >= 0 and int(ids.max()) < experts
    assert all(len(set(row)) == top for row in ids.tolist())
    assert bool(results[1][1][1::8].isnan().all())
