"""Norm, rotation and cache write of rows whose parts are whole pieces of four elements, in both block sizes (by the row's width):
against the same in 64 bits, and against the kernel for rows of any kind."""

import pytest
import torch

from test_gpu_routed_wide import rand

pytestmark = pytest.mark.gpu


def rotated(x, positions, inv_freq, dims, magnitude, interleaved):
    angle = positions.double().view(-1, 1, 1) * inv_freq.double()
    cos, sin = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude
    first, second = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    out[..., first] = x[..., first] * cos - x[..., second] * sin
    out[..., second] = x[..., second] * cos + x[..., first] * sin
    return out


@pytest.mark.parametrize("tokens,heads,kv_heads,dim,vdim", [
    (3, 2, 1, 4, 8), (400, 4, 2, 64, 64), (5, 16, 2, 128, 128), (300, 33, 1, 128, 60), (400, 60, 4, 128, 64)])
@pytest.mark.parametrize("norm,v_norm,bias,interleaved,rot", [
    (1, 0, False, False, 1), (0, 1, True, True, 1), (1, 1, True, False, 0), (0, 0, False, False, 1)])
def test_rows_in_pieces(tokens, heads, kv_heads, dim, vdim, norm, v_norm, bias, interleaved, rot):
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    ops = Runtime("cuda:0", "float32").ops
    ops._load_streams()
    page_size, eps, magnitude = 16, 1e-6, 1.25
    rot_dims = max(dim // 2 // 8 * 8, 4 if interleaved else 0) * rot
    q_width, k_width, v_width = heads * dim, kv_heads * dim, kv_heads * vdim
    width = q_width + k_width + v_width
    src = rand(tokens, width + 4, seed=1)
    gains = [1 + rand(n, seed=s, scale=0.2) for n, s in ((q_width, 2), (k_width, 3))]
    shift = rand(width, seed=4)
    positions = (torch.arange(tokens) * 7 % (tokens + 40)).int()
    pages = -(-(tokens + 40) // page_size)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(5)).int().view(1, -1)
    freq = 10000.0 ** (-torch.arange(rot_dims // 2) / max(rot_dims // 2, 1)) if rot_dims else None
    k_pool = torch.full((pages, kv_heads, page_size, dim), 7.0).cuda()
    v_pool = torch.full((pages, kv_heads, page_size, vdim), 7.0).cuda()
    out = torch.full((tokens + 1, q_width + 4), 7.0).cuda()
    on = [t.cuda() if t is not None else None for t in (src, shift if bias else None, positions, table, *gains, freq)]
    pointer = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
    requests = torch.zeros(tokens, dtype=torch.int32).cuda()
    ops._norm_kv_write(pointer(on[0]), pointer(on[1]), out.data_ptr(), q_width + 4, pointer(on[2]), requests.data_ptr(),
                       pointer(on[3]), pages, pages, k_pool.data_ptr(), v_pool.data_ptr(), pointer(on[4]), pointer(on[5]),
                       tokens, heads, kv_heads, dim, vdim, page_size, norm, v_norm, eps, 1, width + 4, 0, pointer(on[6]),
                       rot_dims, magnitude, int(interleaved), None, 0.0, 0, None, 0, None, None, 0, ops.error_word.data_ptr(),
                       ops.stream)
    ops.check_errors()
    x = src[:, :width].double() + (shift.double() if bias else 0)
    q, k, v = x[:, :q_width], x[:, q_width:q_width + k_width], x[:, q_width + k_width:].view(tokens, kv_heads, vdim)
    if norm:
        q, k = (t / torch.sqrt((t * t).mean(1, keepdim=True) + eps) * g.double() for t, g in ((q, gains[0]), (k, gains[1])))
    q, k = q.view(tokens, heads, dim), k.view(tokens, kv_heads, dim)
    if rot_dims:
        q, k = (rotated(t, positions, freq, rot_dims, magnitude, interleaved) for t in (q, k))
    if v_norm:
        v = v / torch.sqrt((v * v).mean(2, keepdim=True) + eps)
    page, place = table[0][positions.long() // page_size].long(), positions.long() % page_size
    got = out.cpu().double()
    # products and sums of float32; an angle of up to 440 is off by half a unit of its last place, 1.5e-5
    assert float((got[:tokens, :q_width] - q.reshape(tokens, -1)).abs().max()) < 2e-4
    assert float((got[tokens:] - 7).abs().max()) == 0 and float((got[:, q_width:] - 7).abs().max()) == 0
    last = {int(p): t for t, p in enumerate(positions)}      # a position that comes twice: either row may win
    single = torch.tensor([t for p, t in last.items() if int((positions == p).sum()) == 1])
    assert float((k_pool.cpu()[page, :, place].double() - k)[single].abs().max()) < 2e-4
    assert float((v_pool.cpu()[page, :, place].double() - v)[single].abs().max()) < 2e-5


def write_rows(ops, src, positions, requests, table, heads, kv_heads, dim, pools, norm=None, freq=None, extra=(None, 0.0, 0), active=None,
               write=1, magnitude=1.25):
    """One call with rows of ``src`` (a view of columns: its stride decides which kernel runs); q, and the pools are written."""
    tokens, q_width = src.shape[0], heads * dim
    pages = pools[0].shape[0] if pools else 0
    out = torch.full((tokens, q_width), 7.0, dtype=ops.dtype).cuda()
    pointer = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
    held = [pointer(t) for t in (pools or (None, None))]
    q_gain, k_gain = norm or (None, None)
    ops._norm_kv_write(src.data_ptr(), None, out.data_ptr(), q_width, positions.data_ptr(), pointer(requests), pointer(table),
                       table.shape[1] if table is not None else 0, pages, *held, pointer(q_gain), pointer(k_gain), tokens, heads,
                       kv_heads, dim, dim, 16, int(norm is not None), 0, 1e-6, write, src.stride(0), ops._code_of(src), pointer(freq),
                       0 if freq is None else 2 * freq.numel(), magnitude, 0, pointer(extra[0]), extra[1], extra[2], None, 0, None,
                       pointer(active), ops._code_of(out), ops.error_word.data_ptr(), ops.stream)
    return out


@pytest.mark.parametrize("shift", [0, 1])          # rows in pieces, and rows of any kind
def test_queries_alone_need_no_pages(shift):
    """A call that writes nothing to the cache reads no table and no requests."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    ops = Runtime("cuda:0", "float32").ops
    ops._load_streams()
    tokens, heads, dim = 5, 4, 64
    src = rand(tokens, 6 * dim + 4 + shift, seed=1).cuda()
    positions = torch.arange(tokens, dtype=torch.int32).cuda() * 9
    q = write_rows(ops, src, positions, None, None, heads, 1, dim, None, write=0)
    ops.check_errors()
    assert torch.equal(q, src[:, :heads * dim])


@pytest.mark.parametrize("heads,kv_heads", [(16, 2), (40, 4)])          # blocks of 256 threads and of 512
@pytest.mark.parametrize("source", ["float32", "bfloat16"])
@pytest.mark.parametrize("norm", [False, True])
def test_rows_in_pieces_as_rows_of_any_kind(heads, kv_heads, source, norm):
    """bfloat16 queries and pages, factors a head, factors by position, a request that only pads and one whose page is missing:
    the kernel for pieces writes what the other one writes (which an odd stride asks for), and leaves alone what it leaves."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime
    from cloud_inference_from_scratch_b200.native.ops import KernelError

    ops = Runtime("cuda:0", "bfloat16").ops
    ops._load_streams()
    tokens, dim, page_size = 48, 128, 16
    width = (heads + 2 * kv_heads) * dim
    rows = rand(tokens, width, seed=1).to(getattr(torch, source))
    requests = (torch.arange(tokens) // 12).int().cuda()               # four of twelve tokens
    positions = (torch.arange(tokens) % 12 + 10).int().cuda()          # over two pages each
    table = torch.tensor([[0, 1], [2, 3], [4, -1], [6, 7]], dtype=torch.int32).cuda()
    active = torch.tensor([1, 0, 1, 1], dtype=torch.int32).cuda()
    factors, freq = (1 + rand(heads, seed=2, scale=0.3)).cuda(), (10000.0 ** (-torch.arange(32) / 32)).cuda()
    gains = [(1 + rand(n * dim, seed=s, scale=0.2)).cuda() for n, s in ((heads, 3), (kv_heads, 4))] if norm else None
    results = []
    for extra in (4, 3):          # columns behind the row
        src = torch.zeros(tokens, width + extra, dtype=rows.dtype).cuda()
        src[:, :width] = rows.cuda()
        pools = [torch.full((8, kv_heads, page_size, dim), 7.0, dtype=torch.bfloat16).cuda() for _ in range(2)]
        q = write_rows(ops, src, positions, requests, table, heads, kv_heads, dim, pools, gains, freq, (factors, 0.4, 4), active)
        with pytest.raises(KernelError, match="no valid cache page"):
            ops.check_errors()
        ops.check_errors()
        results.append([t.float().cpu() for t in (q, *pools)])
    for pieces, plain in zip(*results):
        # float32 sums in another order, rounded to bfloat16: a unit of its last place where a value is near the middle of two
        assert float((pieces - plain).abs().max()) <= 2.0 ** -7 * float(plain.abs().max())
        assert float((pieces != plain).float().mean()) < 1e-2
    k, v = results[0][1:]
    for pool in (k, v):
        assert bool((pool[2:4] == 7).all()) and bool((pool[5] == 7).all())          # the request that pads; no page
        assert bool((pool[0, :, 10:] != 7).all()) and bool((pool[1, :, :6] != 7).all()) and bool((pool[4, :, 10:] != 7).all())
        assert bool((pool[0, :, :10] == 7).all()) and bool((pool[1, :, 6:] == 7).all()) and bool((pool[4, :, :10] == 7).all())
