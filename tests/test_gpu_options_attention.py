"""The kernels for layers with options (windows, kept keys, penalties, caps, slopes, sinks, gates): prompt portions on tcgen05, against
plain attention in 64 bits and against the mma.sync kernel, which computes the same for other sizes; single tokens on the
split decode kernel."""

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

OPTIONS = [
    dict(),
    dict(window=64, penalty=True),
    dict(window=130, keep=3, sink=True),
    dict(window=257, keep=140, gates=True, slopes=True),
    dict(cap=5.0, sink=True, gates=True),
    dict(window=1, keep=20),
    dict(negative=True),
]


def rand(*shape, seed, scale=1.0):
    generator = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=generator) * scale


def nobodys_pages(*shape):
    """What pages hold that no request has, and the rows of a page behind a request's last key: whatever a former owner left,
    overflows among it."""
    pool = torch.full(shape, math.nan)
    pool[1::3], pool[2::3] = math.inf, 100.0
    return pool.bfloat16()


def oracle(q, k, v, position, group, scale, o, heads):
    """One token's rows [heads, dim] over keys [.., kv, dim] of positions 0 .. position."""
    out = torch.empty(heads, v.shape[2], dtype=torch.float64)
    gap = position - torch.arange(position + 1, dtype=torch.float64)
    seen = torch.ones(position + 1, dtype=torch.bool)
    if o.window:
        seen = (gap < o.window) | (torch.arange(position + 1) < o.keep)
    for h in range(heads):
        s = (k[:position + 1, h // group] @ q[h]) * scale
        if o.cap:
            s = o.cap * torch.tanh(s / o.cap)
        if o.slopes is not None:
            s = s - o.slopes[h] * gap
        if o.penalty is not None:
            s = s - o.penalty[0][h] * torch.log1p(o.penalty[1][h] * gap)
        s = s.masked_fill(~seen, -math.inf)
        if o.sinks is not None:
            s = torch.cat([s, o.sinks[h].double().view(1)])
        out[h] = torch.softmax(s, 0)[:position + 1] @ v[:position + 1, h // group]
    return out


@pytest.mark.parametrize("dim,kv_heads,group,page", [(128, 2, 8, 16), (64, 1, 3, 48), (128, 1, 1, 256), (64, 2, 16, 128)])
@pytest.mark.parametrize("option", range(len(OPTIONS)))
def test_portions_with_options(option, dim, kv_heads, group, page):
    """Requests that begin, that go on over a long context, that end at and beside tile edges, and a single token in
    front; pages in descending order for some requests and in a row for others, gone where a window has left them behind.  A
    weight enters as two bfloat16 terms and the result is rounded once: 2^-9 of a row's largest value, and as much again
    for the exponentials' own error under the largest scores."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime
    from cloud_inference_from_scratch_b200.native.tensor_attention import plan_tiles

    ops = Runtime("cuda:0", "bfloat16").ops
    ops.require_portion_attention(dim)
    fast = ops._tensor_attention[dim]
    assert fast._prompt_options is not None
    asked = OPTIONS[option]
    heads = kv_heads * group
    lengths, contexts = [1, 40, 17, 2, 129], [5, 0, 300, 126, 511]
    count, tokens = len(lengths), sum(lengths)
    scale = (-1 if asked.get("negative") else 1) * dim ** -0.5
    o = SimpleNamespace(window=asked.get("window", 0), keep=asked.get("keep", 0), cap=asked.get("cap", 0.0), slopes=None,
                        penalty=None, sinks=None, gates=None)
    if asked.get("slopes"):
        o.slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)])
    if asked.get("penalty"):
        o.penalty = (rand(heads, seed=1).abs(), rand(heads, seed=2).abs())
    if asked.get("sink"):
        o.sinks = rand(heads, seed=3)
    if asked.get("gates"):
        o.gates = rand(tokens, heads + 1, seed=4)
    width = -(-max(c + n for c, n in zip(contexts, lengths)) // page)
    table = torch.full((count, width), -1, dtype=torch.int32)
    pools = [nobodys_pages(count * width, kv_heads, page, dim) for _ in range(2)]
    keys, values = [], []
    for r in range(count):
        total = contexts[r] + lengths[r]
        k, v = rand(total, kv_heads, dim, seed=10 + r, scale=1.5).bfloat16(), rand(total, kv_heads, dim, seed=20 + r).bfloat16()
        keys.append(k.double()), values.append(v.double())
        lowest = max(0, contexts[r] - o.window + 1) if o.window else 0
        for index in range(-(-total // page)):
            if (index + 1) * page <= lowest and index * page >= o.keep:
                continue                                        # behind the window
            table[r, index] = r * width + (index if r % 2 else width - 1 - index)
            rows = slice(index * page, min((index + 1) * page, total))
            for pool, source in zip(pools, (k, v)):
                pool[table[r, index], :, :rows.stop - rows.start] = source[rows].transpose(0, 1)
    q = rand(tokens, heads * dim, seed=6, scale=1.5).bfloat16()
    starts = np.cumsum([0, *lengths]).astype(np.int32)
    lens = np.asarray(lengths, dtype=np.int32)
    as_int = lambda numbers: torch.tensor(numbers, dtype=torch.int32).cuda()  # noqa: E731
    pools = [pool.cuda() for pool in pools]
    kv = SimpleNamespace(group=0, k=pools[0], v=pools[1], num_pages=count * width, page_size=page)
    ctx = SimpleNamespace(block_tables=[table.cuda()], context_lens=as_int(contexts), query_lens=as_int(lengths),
                          query_start=torch.from_numpy(starts).cuda(), num_single=1, num_requests=count)
    plan = {name: torch.from_numpy(array).cuda() for name, array in plan_tiles(lens, group, skip=1).items()}
    device = lambda t: None if t is None else t.cuda()  # noqa: E731
    gates, sinks, slopes = device(o.gates), device(o.sinks), device(o.slopes)
    penalty = None if o.penalty is None else tuple(device(t) for t in o.penalty)
    results = []
    for kernel in (fast._prompt_options, None):
        held, fast._prompt_options = fast._prompt_options, kernel
        out = torch.full((tokens, heads * dim), 7.0, dtype=torch.bfloat16).cuda()
        fast.run_portions(q.cuda(), out, ctx, kv, heads, kv_heads, scale, o.window, plan, penalty, True, keep_first=o.keep,
                          sinks=sinks, softcap=o.cap, slopes=slopes, gates=None if gates is None else gates[:, 1:])
        fast._prompt_options = held
        ops.check_errors()
        results.append(out.float().cpu())
    assert float((results[0][0] - 7.0).abs().max()) == 0        # the single token is another kernel's
    row = 0
    for r in range(count):
        for t in range(lengths[r]):
            if r > 0 and (t < 2 or t > lengths[r] - 3 or t % 16 in (0, 15)):
                want = oracle(q[row].double().view(heads, dim), keys[r], values[r], contexts[r] + t, group, scale, o, heads)
                if o.gates is not None:
                    want = want * torch.sigmoid(o.gates[row, 1:].double()).view(-1, 1)
                got = results[0][row].view(heads, dim).double()
                bound = 2.0 ** -8 * float(want.abs().max()) + 1e-6
                assert float((got - want).abs().max()) <= bound, (r, t)
            row += 1
    assert torch.allclose(results[0], results[1], rtol=2.0 ** -7, atol=2.0 ** -8)


@pytest.mark.parametrize("dim,kv_heads,group,page", [(128, 2, 8, 16), (64, 1, 3, 32), (192, 1, 16, 16), (128, 1, 20, 128), (256, 2, 1, 64)])
@pytest.mark.parametrize("option", [0, 1, 4, 6, 7])
def test_single_tokens_with_options(option, dim, kv_heads, group, page):
    """First tokens, contexts at and beside the edges of blocks and ranges, one that many CTAs share; pages in descending
    order, gone behind a window.  The weights enter whole, the result is rounded once."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    ops = Runtime("cuda:0", "bfloat16").ops
    ops.require_portion_attention(dim)
    fast = ops._tensor_attention[dim]
    asked = (OPTIONS + [dict(window=300, slopes=True, gates=True, penalty=True, cap=3.0)])[option]
    heads = kv_heads * group
    contexts = [0, 15, 16, 63, 64, 300, 2100]
    count, total_keys = len(contexts), max(contexts) + 1
    scale = (-1 if asked.get("negative") else 1) * dim ** -0.5
    o = SimpleNamespace(window=asked.get("window", 0), keep=0, cap=asked.get("cap", 0.0), slopes=None, penalty=None,
                        sinks=rand(heads, seed=3) if asked.get("sink") else None,
                        gates=rand(count, heads + 1, seed=4) if asked.get("gates") else None)
    if asked.get("slopes"):
        o.slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)])
    if asked.get("penalty"):
        o.penalty = (rand(heads, seed=1).abs(), rand(heads, seed=2).abs())
    width = -(-total_keys // page)
    table = torch.full((count, width), -1, dtype=torch.int32)
    pools = [nobodys_pages(count * width, kv_heads, page, dim) for _ in range(2)]
    keys, values = [], []
    for r, context in enumerate(contexts):
        k, v = rand(context + 1, kv_heads, dim, seed=10 + r, scale=1.5).bfloat16(), rand(context + 1, kv_heads, dim, seed=30 + r).bfloat16()
        keys.append(k.double()), values.append(v.double())
        lowest = max(0, context - o.window + 1) if o.window else 0
        for index in range(lowest // page, -(-(context + 1) // page)):
            table[r, index] = r * width + width - 1 - index
            rows = slice(index * page, min((index + 1) * page, context + 1))
            for pool, source in zip(pools, (k, v)):
                pool[table[r, index], :, :rows.stop - rows.start] = source[rows].transpose(0, 1)
    q = rand(count, heads * dim, seed=6, scale=1.5).bfloat16()
    pools = [pool.cuda() for pool in pools]
    kv = SimpleNamespace(group=0, k=pools[0], v=pools[1], num_pages=count * width, page_size=page)
    ctx = SimpleNamespace(block_tables=[table.cuda()], context_lens=torch.tensor(contexts, dtype=torch.int32).cuda())
    assert fast.splits_decode(kv)
    device = lambda t: None if t is None else t.cuda()  # noqa: E731
    gates, sinks, slopes = device(o.gates), device(o.sinks), device(o.slopes)
    penalty = None if o.penalty is None else tuple(device(t) for t in o.penalty)
    out = torch.full((count + 1, heads * dim), 7.0, dtype=torch.bfloat16).cuda()
    fast.run_singles(q.cuda(), out, ctx, kv, count, heads, kv_heads, scale, o.window, penalty, sinks=sinks, softcap=o.cap,
                     slopes=slopes, gates=None if gates is None else gates[:, 1:])
    ops.check_errors()
    assert float((out[count] - 7.0).abs().max()) == 0 and int(fast._split_tickets.abs().sum()) == 0
    for r, context in enumerate(contexts):
        want = oracle(q[r].double().view(heads, dim), keys[r], values[r], context, group, scale, o, heads)
        if o.gates is not None:
            want = want * torch.sigmoid(o.gates[r, 1:].double()).view(-1, 1)
        got = out[r].view(heads, dim).double().cpu()
        assert float((got - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-6, r


@pytest.mark.parametrize("option", [2, 1, 4])
def test_a_short_portion_whatever_the_width_of_the_table(option):
    """A table as wide as the longest request of the step, or of the model where graphs are enabled, changes no bit."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime
    from cloud_inference_from_scratch_b200.native.tensor_attention import plan_tiles

    ops = Runtime("cuda:0", "bfloat16").ops
    ops.require_portion_attention(128)
    asked, heads, kv_heads, page, length = OPTIONS[option], 16, 2, 16, 33
    pools = [rand(64, kv_heads, page, 128, seed=s).bfloat16().cuda() for s in (1, 2)]
    kv = SimpleNamespace(group=0, k=pools[0], v=pools[1], num_pages=64, page_size=page)
    q = rand(length, heads * 128, seed=3).bfloat16().cuda()
    penalty = tuple(rand(heads, seed=s).abs().cuda() for s in (4, 5)) if asked.get("penalty") else None
    sinks = rand(heads, seed=6).cuda() if asked.get("sink") else None
    lens = np.asarray([length], dtype=np.int32)
    plan = {name: torch.from_numpy(array).cuda() for name, array in plan_tiles(lens, heads // kv_heads).items()}
    as_int = lambda numbers: torch.tensor(numbers, dtype=torch.int32).cuda()  # noqa: E731
    results = []
    for width in (3, 4, 5, 17, 40):
        ctx = SimpleNamespace(block_tables=[torch.arange(7, 7 + width, dtype=torch.int32).view(1, -1).cuda()], context_lens=as_int([0]),
                              query_lens=as_int([length]), query_start=as_int([0, length]), num_single=0, num_requests=1)
        out = torch.empty_like(q)
        ops._tensor_attention[128].run_portions(q, out, ctx, kv, heads, kv_heads, 128 ** -0.5, asked.get("window", 0), plan, penalty,
                                                True, keep_first=asked.get("keep", 0), sinks=sinks, softcap=asked.get("cap", 0.0))
        results.append(out)
    ops.check_errors()
    assert all(torch.equal(results[0], other) for other in results[1:])


def test_a_larger_step_of_single_tokens_makes_no_memory():
    """The split decode kernel has its own, sized once; a batch and a table that grow behind a captured graph must not ask for
    the group kernel's."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    ops = Runtime("cuda:0", "bfloat16").ops
    ops.require_portion_attention(128)
    page, heads, kv_heads = 16, 16, 2
    pools = [rand(600, kv_heads, page, 128, seed=s).bfloat16().cuda() for s in (1, 2)]
    kv = SimpleNamespace(group=0, k=pools[0], v=pools[1], num_pages=600, page_size=page)
    sinks = rand(heads, seed=3).cuda()
    for requests, width in ((2, 17), (4, 130)):
        q = rand(requests, heads * 128, seed=4).bfloat16().cuda()
        out = torch.empty_like(q)
        as_int = lambda numbers: torch.tensor(numbers, dtype=torch.int32).cuda()  # noqa: E731
        contexts = [page * width - 1 - r for r in range(requests)]
        table = torch.arange(requests * width, dtype=torch.int32).view(requests, width).cuda()
        ctx = SimpleNamespace(block_tables=[table], context_lens=as_int(contexts), positions=as_int(contexts),
                              request_of_token=as_int(list(range(requests))), num_single=requests, num_requests=requests)
        ops.attention_penalised(q, out, ctx, kv, heads, kv_heads, 128, 128, 128 ** -0.5, 0, None, sinks=sinks)
        ops.check_errors()
        if width == 17:
            generation = ops.scratch_generation
            ops.freeze_scratch()
    assert ops.scratch_generation == generation


@pytest.mark.parametrize("options", [False, True])
def test_what_one_object_asks_the_device_takes_nothing_from_another(options):
    """The shared memory that launches may ask for belongs to the kernel: an object with fewer head rows on a kv head, which
    asks what rings fit, must not lower it."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime
    from test_gpu_kernels import tensor_case

    one = {torch.bfloat16: Runtime("cuda:0", "bfloat16").ops}

    def decode():
        if options:
            test_single_tokens_with_options(1, 128, 1, 20, 128)
        else:
            tensor_case(one, 128, [3000, 77], [1, 1], 16, 1, 128, 16, seed=1)

    decode()
    other = Runtime("cuda:0", "bfloat16").ops
    other.require_portion_attention(128)
    other._tensor_attention[128].split_choices(1, options)
    decode()
