"""Float32 products on the tensor cores: three bfloat16 terms a value, sums taken out every 128 columns."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def rand(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


@pytest.fixture(scope="module")
def ops():
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    return Runtime("cuda:0", "float32").ops


def product(ops, x, w, bias, columns=0):
    """With a row behind the result that has to stay as it is."""
    m, n = x.shape[0], w.shape[0]
    out = torch.full((m + 1, n), 7.0).cuda()
    ops._gemm_f32(x.data_ptr(), w.data_ptr(), None if bias is None else bias.data_ptr(), out.data_ptr(), m, n, x.shape[1],
                  columns, ops.error_word.data_ptr(), ops.stream)
    ops.check_errors()
    assert float((out[m] - 7.0).abs().max()) == 0
    return out[:m]


@pytest.mark.parametrize("n", [1, 31, 64, 65, 130])
@pytest.mark.parametrize("k", [512, 516, 640, 1100, 2052])
def test_rows_columns_and_steps_that_end_inside_a_tile(ops, n, k):
    """An accumulator takes 8 cut additions of 2^-23 an interval, every interval's sum is rounded once (2^-24), the pairs
    left out are three of 2^-26: of the sum of the products' magnitudes.  Tiles and the number of rows change no bit."""
    bias = rand(n, seed=3).cuda()
    for m in (1, 33, 128, 129, 300):
        x, w = rand(m, k, seed=m).cuda(), rand(n, k, seed=m + 1).cuda()
        out = product(ops, x, w, bias, 64)
        assert torch.equal(out, product(ops, x, w, bias, 32))
        assert torch.equal(out[-1:], product(ops, x[-1:].contiguous(), w, bias))
        bound = 8 * 2.0 ** -23 + (k // 128 + 2) * 2.0 ** -24 + 3 * 2.0 ** -26
        magnitude = x.double().abs() @ w.double().abs().T + bias.double().abs()
        assert bool(((out.double() - x.double() @ w.double().T - bias.double()).abs() <= bound * magnitude).all())


def test_many_tiles_a_block_and_rows_that_are_not_finite(ops):
    """More tiles than blocks.  Rows and columns with an infinity, a NaN or a value beyond bfloat16's largest are summed in
    float32 in ascending order, whatever their neighbours hold, and nothing of them reaches other rows."""
    m, n, k = 290, 8200, 516
    x, w = rand(m, k, seed=1), rand(n, k, seed=2)
    clean = product(ops, x.cuda(), w.cuda(), None)
    x[3, 5], x[130, 9], x[289, 515], w[20, 1], w[8199, 3], w[4097, 0] = float("inf"), float("nan"), 3.4e38, -float("inf"), float("nan"), -3.4e38
    x, w = x.cuda(), w.cuda()
    out, plain = product(ops, x, w, None), torch.empty(m, n).cuda()
    ops._gemm_simt(x.data_ptr(), w.data_ptr(), None, plain.data_ptr(), m, n, k, 0, 0, 0, ops.stream)
    apart = torch.zeros(m, n, dtype=torch.bool)
    apart[[3, 130, 289]] = True
    apart[:, [20, 8199, 4097]] = True
    assert torch.equal(out.cpu()[apart].nan_to_num(7.0), plain.cpu()[apart].nan_to_num(7.0))
    assert torch.equal(out.cpu()[~apart], clean.cpu()[~apart])


def test_the_runtime_sends_long_aligned_rows_there(ops):
    for k, there in ((512, True), (508, False), (514, False)):
        x, w = rand(5, k, seed=1).cuda(), rand(9, k, seed=2).cuda()
        out = ops.linear(x, w, None, torch.empty(5, 9).cuda())
        few = ops.linear(x, w, None, torch.empty(5, 9).cuda(), few_rows=True)
        assert torch.equal(few[:1], ops.linear(x[:1].contiguous(), w, None, torch.empty(1, 9).cuda(), few_rows=True))
        assert torch.equal(out, few) != there
        assert torch.equal(out, product(ops, x, w, None)) if there else not ops._gemm_f32_takes(x.data_ptr(), w.data_ptr(), k)
        assert float((out.double() - x.double() @ w.double().T).abs().max()) <= 1e-4
