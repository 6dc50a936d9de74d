"""Attention beside rows of the cache that are not the request's: pages that nobody has, the tail of a request's last page,
another request's values.  They may hold infinities and NaN; a result must not know of them."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

import test_gpu_bozevik
import test_gpu_kernels
import test_gpu_program

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.fixture
def foreign(monkeypatch):
    """The pools that the attention cases build, with every row that no request owns overflowed."""
    plain = test_gpu_kernels.paged_setup

    def setup(lengths, page, heads, dim, dtype, **kwargs):
        k_pool, v_pool, table, dense, total = plain(lengths, page, heads, dim, dtype, **kwargs)
        mine = torch.zeros(total, page, dtype=torch.bool)
        for r, n in enumerate(lengths):
            for p in range(-(-n // page)):
                mine[int(table[r, p]), :min(page, n - p * page)] = True
        left = torch.full((total, page), float("nan"))
        left[:, 1::3], left[:, 2::3] = float("inf"), -float("inf")
        for pool in (k_pool, v_pool):
            rows = pool.transpose(1, 2)
            rows[~mine.cuda()] = left[~mine].to(dtype).cuda().view(-1, 1, 1).expand(-1, heads, dim)
        return k_pool, v_pool, table, dense, total

    monkeypatch.setattr(test_gpu_kernels, "paged_setup", setup)


@pytest.fixture(scope="module")
def ops():
    from cloud_inference_from_scratch_b200.native import Ops

    made = {BF16: Ops("cuda:0", BF16)}
    yield made
    made[BF16].check_errors()


@pytest.mark.parametrize("pages", ["shuffled", "consecutive", "runs"])
@pytest.mark.parametrize("dim,page,q_heads,kv_heads", [(128, 16, 16, 2), (64, 48, 7, 1), (128, 256, 3, 3), (64, 16, 20, 1)])
def test_prompt_portions(ops, foreign, dim, page, q_heads, kv_heads, pages):
    """Portions that end inside a key tile, at its edge and one key behind it; long contexts, whose keys go to several CTAs."""
    test_gpu_kernels.tensor_case(ops, dim, [0, 127, 128, 300, 0], [129, 2, 256, 77, 1], q_heads, kv_heads, dim, page, seed=1, pages=pages)
    test_gpu_kernels.tensor_case(ops, dim, [3000, 17], [40, 5], q_heads, kv_heads, dim, page, seed=2, pages=pages)


@pytest.mark.parametrize("dim,page,q_heads,kv_heads,window", [(128, 16, 16, 2, 0), (64, 32, 20, 1, 0), (192, 16, 3, 1, 0), (256, 64, 2, 1, 0),
                                                              (128, 16, 16, 2, 100), (32, 8, 4, 2, 0), (32, 8, 4, 2, 37)])
def test_single_tokens(ops, foreign, dim, page, q_heads, kv_heads, window):
    contexts = [0, 15, 16, 63, 64, 300, 2100]
    test_gpu_kernels.tensor_case(ops, dim, contexts, [1] * len(contexts), q_heads, kv_heads, dim, page, window=window, seed=3)


@pytest.mark.parametrize("dim,page,window", [(128, 16, 0), (64, 32, 33), (128, 64, 1000)])
def test_single_tokens_of_a_recorded_program(ops, foreign, dim, page, window):
    test_gpu_program.program_attention(ops[BF16], dim, [0, 15, 16, 63, 64, 300, 2100], 8, 2, page, window=window, seed=4)


@pytest.mark.parametrize("window", [0, 130])
@pytest.mark.parametrize("dim,rot,vdim,rank", [(128, 64, 128, 96), (40, 16, 72, 24)])
def test_expanded_latents_of_a_neighbour(window, dim, rot, vdim, rank):
    """The portions' expanded rows lie one after the other: the last tile of one holds the next one's first rows."""
    heads, page = 2, 16
    lengths, contexts = [150, 40, 129], [20, 300, 0]
    total = [a + b for a, b in zip(lengths, contexts)]
    rt = test_gpu_bozevik.runtime("bfloat16")
    rand = test_gpu_bozevik.rand
    rotation = SimpleNamespace(inv_freq=torch.ones(rot // 2).cuda(), magnitude=1.0, interleaved=True, dims=rot)
    q = rand(sum(lengths), heads * (dim + rot), seed=1)
    w_kv = rand(heads * (dim + vdim), rank, scale=rank ** -0.5, seed=2).bfloat16().cuda()
    results = []
    for broken in (False, True):
        c = [rand(t, rank, seed=20 + i).bfloat16() for i, t in enumerate(total)]
        if broken:
            c[1][:] = float("inf")
        r = [rand(t, rot, seed=30 + i).bfloat16() for i, t in enumerate(total)]
        ctx, kv = test_gpu_bozevik.paged(c, r, contexts, lengths, page, BF16, seed=0)
        plan = {name: torch.from_numpy(array).cuda() for name, array in rt.ops.plan_latent_prompt(ctx.host, window).items()}
        out = torch.full((sum(lengths), heads * vdim), 5.0, dtype=BF16).cuda()
        rt.ops.latent_prompt(q.cuda(), out, ctx, kv, rotation, plan, w_kv, None, heads, dim, rot, vdim, rank, 0.2, window=window)
        rt.ops.check_errors()
        results.append(out.float().cpu())
    at = np.cumsum([0, *lengths])
    for i in (0, 2):
        assert torch.equal(results[0][at[i]:at[i + 1]], results[1][at[i]:at[i + 1]])
    assert not bool(results[1][at[1]:at[2]].isfinite().any())      # the request that overflowed sees that
