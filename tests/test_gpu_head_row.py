"""The head for one token row: odd and single table rows, rows of one unit, of a remainder behind whole turns of a warp, of many turns. Against 64 bits: a
lane adds ceil(cols / 256) * 8 products in a row and a warp the lanes' sums in five steps, so the error is at most that many roundings of sum |x w|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 33, 4737, 9473])
@pytest.mark.parametrize("cols", [8, 264, 1280, 1288, 2560, 4096, 14520])
def test_one_row(ctx, rows, cols):
    import torch
    from lemonade_burn_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    w = torch.randn(rows, cols, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(1, cols, generator=g, device="cuda")
    got = ops.bf16_linear(x, w, ctx).double()
    want = x.double() @ w.double().T
    bound = (-(-cols // 256) * 8 + 5) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((got - want).abs() <= bound).all())
    ctx.check_device_error()
