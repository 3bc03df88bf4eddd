"""Gate and up in one GEMM whose epilogue forms relu(gate)^2 * up: the bits of the two projections followed by lbk_relu2_mul, around the tile of 64 pairs of
rows, ragged token tiles of both forms, K of one block to a ragged stage."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 128), (63, 640), (64, 896), (65, 256), (700, 2560), (6912, 384)])
@pytest.mark.parametrize("m", [1, 9, 64, 65, 193, 400])
def test_bits_of_the_separate_operations(oracle, ctx, rows, cols, m):
    import torch
    from lemonade_burn_b200 import _lib, ops
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(rows + cols + m)
    lins = [ops.TernaryLinear(torch.from_numpy(oracle.pack_matrix(rng.choice(np.array([-1, 0, 1], dtype=np.int8), size=(rows, cols), p=[0.3, 0.4, 0.3]))).cuda(),
                              50.0 + 7 * i, cols, ctx) for i in range(2)]
    x = torch.from_numpy(rng.standard_normal((m, cols)).astype(np.float32)).cuda()
    q = torch.zeros(m, -(-cols // 128) * 128, dtype=torch.int8, device="cuda")
    s, t = torch.zeros(m, device="cuda"), torch.zeros(m, dtype=torch.int32, device="cuda")
    _lib.check(lib.lbk_quantize_acts_dev(ctx.handle, x.data_ptr(), m, cols, q.data_ptr(), s.data_ptr(), t.data_ptr(), st))
    gate, up = ops.ternary_gemm_q(q, s, t, m, lins)
    want, got = torch.empty_like(gate), torch.full_like(gate, float("nan"))
    _lib.check(lib.lbk_relu2_mul(ctx.handle, gate.data_ptr(), up.data_ptr(), gate.numel(), want.data_ptr(), st))
    _lib.check(lib.lbk_ternary_relu2_gemm_dev(ctx.handle, lins[0].weight.handle, lins[1].weight.handle, q.data_ptr(), s.data_ptr(), t.data_ptr(), m, got.data_ptr(), st))
    assert torch.equal(got, want)
    ctx.check_device_error()


def test_matrices_that_do_not_pair_are_refused(oracle, ctx):
    import torch
    from lemonade_burn_b200 import _lib, ops
    lins = [ops.TernaryLinear(torch.zeros(r, 32, dtype=torch.uint8, device="cuda"), 1.0, 128, ctx) for r in (16, 32)]
    b = torch.zeros(4096, device="cuda")
    with pytest.raises(_lib.LbkError):
        _lib.check(_lib.load().lbk_ternary_relu2_gemm_dev(ctx.handle, lins[0].weight.handle, lins[1].weight.handle, b.data_ptr(), b.data_ptr(), b.data_ptr(), 2, b.data_ptr(), 0))
    with pytest.raises(_lib.LbkError):
        _lib.check(_lib.load().lbk_ternary_relu2_gemm_dev(ctx.handle, lins[0].weight.handle, lins[0].weight.handle, None, b.data_ptr(), b.data_ptr(), 2, b.data_ptr(), 0))


@pytest.mark.parametrize("m", [9, 200])
def test_scales_that_are_no_numbers(oracle, ctx, m):
    """Rows whose scale is infinite, no number, zero, below zero or so small that the factors overflow: infinities, NaN and 0 * infinity in the places where the
    separate operations have them."""
    import torch
    from lemonade_burn_b200 import _lib, ops
    lib, st, rows, cols = _lib.load(), torch.cuda.current_stream().cuda_stream, 130, 640
    rng = np.random.default_rng(m)
    lins = [ops.TernaryLinear(torch.from_numpy(oracle.pack_matrix(rng.choice(np.array([-1, 0, 1], dtype=np.int8), size=(rows, cols), p=[0.3, 0.4, 0.3]))).cuda(),
                              50.0 + 7 * i, cols, ctx) for i in range(2)]
    q = torch.from_numpy(rng.integers(-127, 128, (m, cols)).astype(np.int8)).cuda()
    q[1] = 0  # dots of 0 beside infinite factors
    t = q.int().sum(1, dtype=torch.int32)
    s = torch.full((m,), 30.0, device="cuda")
    s[:8] = torch.tensor([float("inf"), 0.0, float("nan"), 0.0, -3.0, 1e-38, 1e-20, float("-inf")], device="cuda")
    s[m - 1] = float("nan")
    gate, up = ops.ternary_gemm_q(q, s, t, m, lins)
    want, got = torch.empty_like(gate), torch.full_like(gate, 7.0)
    _lib.check(lib.lbk_relu2_mul(ctx.handle, gate.data_ptr(), up.data_ptr(), gate.numel(), want.data_ptr(), st))
    _lib.check(lib.lbk_ternary_relu2_gemm_dev(ctx.handle, lins[0].weight.handle, lins[1].weight.handle, q.data_ptr(), s.data_ptr(), t.data_ptr(), m, got.data_ptr(), st))
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and bool(torch.isnan(want).any()) and bool(torch.isinf(want).any())
    assert torch.equal(torch.nan_to_num(got, nan=1.0), torch.nan_to_num(want, nan=1.0))
    ctx.check_device_error()
