"""Float32 products whose rows do not all fit the scratch memory of their terms."""

import pytest
import torch

from test_gpu_f32_products import rand

pytestmark = pytest.mark.gpu


def test_rows_in_blocks_change_no_bit(monkeypatch):
    """More rows than a block, and scratch memory that may not grow: blocks of what it holds."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime
    from cloud_inference_from_scratch_b200.native import ops as module

    ops = Runtime("cuda:0", "float32").ops
    m, n, k = 300, 130, 1100
    x, w = rand(m, k, seed=1).cuda(), rand(n, k, seed=2).cuda()
    x[7, 3] = float("nan")
    want = ops.linear(x, w, None, torch.empty(m, n).cuda())
    monkeypatch.setattr(module, "F32_BLOCK", 77)
    assert torch.equal(ops.linear(x, w, None, torch.empty(m, n).cuda()).nan_to_num(7.0), want.nan_to_num(7.0))
    frozen = Runtime("cuda:0", "float32").ops
    frozen._partial_buffers["gemm_f32.terms"] = torch.empty(frozen._gemm_f32_floats(50, k) + 3).cuda()
    frozen.freeze_scratch()
    generation = frozen.scratch_generation
    assert torch.equal(frozen.linear(x, w, None, torch.empty(m, n).cuda()).nan_to_num(7.0), want.nan_to_num(7.0))
    frozen._partial_buffers["gemm_f32.terms"] = torch.empty(9).cuda()
    plain = frozen.linear(x, w, None, torch.empty(m, n).cuda())
    rows = torch.arange(m) != 7
    assert float((plain.cpu()[rows].double() - x.cpu()[rows].double() @ w.cpu().double().T).abs().max()) < 1e-3
    frozen.check_errors()
    assert frozen.scratch_generation == generation
