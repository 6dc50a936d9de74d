"""Scratch memory of the recurrences in chunks: made at first use for every step that the runtime may bring, since it keeps its
place once a captured graph holds it.  No kernel runs here."""

import types
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from cloud_inference_from_scratch_b200.native.ops import BF16, Ops

CHUNK = 32
MAX_ROWS, MAX_REQUESTS = 2048, 16
HEADS, GROUPS, DIM = 16, 8, 4


def ops_of(max_rows=MAX_ROWS, max_requests=MAX_REQUESTS):
    nothing = lambda *args: None  # noqa: E731
    launched = []
    run = lambda *args: launched.append(1)  # noqa: E731
    ops = SimpleNamespace(
        torch=torch, device=torch.device("cpu"), code=BF16, stream=0, launches=0, error_word=None, _partial_buffers={},
        scratch_frozen=False, scratch_generation=0, max_rows=max_rows, max_requests=max_requests, launched=launched,
        mlstm_chunk_tokens=CHUNK, mlstm_chunk_max_dim=128, gla_chunk_tokens=CHUNK, gla_chunk_max_dim=128,
        delta_chunk_tokens=CHUNK, ssd_chunk_tokens=CHUNK, lightning_chunk_tokens=CHUNK,
        # a token's rows and a chunk's sums or states: more of either asks for more
        _mlstm_chunk_floats=lambda tokens, chunks, heads, dim, vdim: 3 * tokens + 50 * chunks,
        _gated_delta_chunk_floats=lambda tokens, chunks, heads, kv_heads, dim, vdim: 3 * tokens + (50 + 9 * kv_heads) * chunks,
        _ssd_chunk_floats=lambda tokens, chunks, heads, groups, dim, vdim: 3 * tokens + 50 * chunks,
        _gla_chunk_floats=lambda chunks, heads, dim: 50 * chunks,
        _delta_lib=SimpleNamespace(handle=SimpleNamespace(cie_delta_chunk_floats=lambda chunks, heads, dim: 50 * chunks)),
        _mlstm_chunked=run, _gated_delta_chunked=run, _ssd_chunked=run, _gla_chunked=run, _delta_chunked=run,
        _lightning_chunked=run, _ssd_scan=nothing, _code_of=lambda t: BF16)
    for name in ("_flush", "_load_recurrent", "_load_ssd", "_load_gla", "_load_delta", "_load_lightning"):
        setattr(ops, name, nothing)
    for name in ("scratch", "freeze_scratch", "_most_chunks"):
        if hasattr(Ops, name):
            setattr(ops, name, types.MethodType(getattr(Ops, name), ops))
    return ops


def step(ops, kind, lengths, kv_heads=GROUPS):
    """One step's call of a recurrence; whether it ran in chunks."""
    tokens = sum(lengths)
    starts = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    host = SimpleNamespace(query_start=starts, query_lens=np.asarray(lengths, dtype=np.int32))
    plan = {name: torch.from_numpy(a) for name, a in Ops._plan_chunks(host, CHUNK).items()}
    ctx = SimpleNamespace(num_requests=len(lengths), query_start=None, slots=None, request_active=None)
    rows, state = torch.zeros(tokens, 1), torch.zeros(1, 1)
    before = len(ops.launched)
    if kind == "mlstm":
        Ops.mlstm_scan(ops, rows, (0,) * 5, None, None, 1.0, 1.0, rows, state, ctx, HEADS, DIM, DIM, plan=plan)
    elif kind == "gated_delta":
        Ops.gated_delta_scan(ops, rows, (0,) * 3, rows, (0, 0), None, None, 1.0, rows, state, ctx, HEADS, kv_heads, DIM, DIM, plan=plan)
    elif kind == "ssd":
        Ops.ssd(ops, rows, (0,) * 3, rows, None, None, None, rows, state, ctx, HEADS, GROUPS, DIM, DIM, plan=plan)
    elif kind == "gla":
        Ops.gla(ops, rows, (0,) * 3, rows, None, 1.0, 1.0, rows, state, ctx, HEADS, DIM, DIM, plan=plan)
    elif kind == "delta":
        Ops.delta_scan(ops, rows, (0,) * 4, rows, None, None, rows, state, ctx, HEADS, DIM, plan=plan)
    else:
        Ops.lightning_chunked(ops, rows, rows, state, None, ctx, plan, HEADS, DIM, DIM)
    return len(ops.launched) > before


KINDS = ["mlstm", "gated_delta", "ssd", "gla", "delta", "lightning"]
UNEVEN = [[230, 270, 250, 262, 240, 281, 250, 265], [2048], [129] * 15 + [113], [2, 3] + [146] * 13 + [145]]


@pytest.mark.parametrize("first", [[40], [256]])
@pytest.mark.parametrize("kind", KINDS)
def test_the_largest_steps_fit_what_a_short_first_prompt_left(kind, first):
    assert all(sum(lengths) == MAX_ROWS and len(lengths) <= MAX_REQUESTS for lengths in UNEVEN[:3])
    ops = ops_of()
    assert step(ops, kind, first)
    ops.freeze_scratch()
    for lengths in UNEVEN:
        assert step(ops, kind, lengths)
    assert ops.scratch_generation == 0


@pytest.mark.parametrize("kind", KINDS)
def test_any_number_of_requests_that_the_runtime_allows_fits(kind):
    """More requests than any fixed allowance: 250 of eight tokens and more, one of a single token behind whole chunks."""
    ops = ops_of(4096, 256)
    assert step(ops, kind, [33])
    ops.freeze_scratch()
    assert step(ops, kind, [8] * 128 + [33] * 93)
    assert step(ops, kind, [16] * 256)


def test_layers_that_share_all_but_the_key_heads_have_scratch_memory_of_their_own():
    ops = ops_of()
    assert step(ops, "gated_delta", [40], kv_heads=1)
    ops.freeze_scratch()
    assert step(ops, "gated_delta", UNEVEN[0], kv_heads=16)
    assert step(ops, "gated_delta", UNEVEN[0], kv_heads=1)
