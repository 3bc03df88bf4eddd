"""The rings of the decode kernels hand a stage back to the copy engine as soon as its words have been multiplied. Many launches behind one another of the
kernels with the shortest stages' lives, the sweep, a projection of few rows and the step in one launch: every result has the bits of the first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _linears(oracle, ctx, cols, rows, seed):
    import torch
    from lemonade_burn_b200 import ops
    rng = np.random.default_rng(seed)
    return [ops.TernaryLinear(torch.from_numpy(oracle.pack_matrix(rng.choice(np.array([-1, 0, 1], dtype=np.int8), size=(r, cols), p=[0.3, 0.4, 0.3]))).cuda(), 50.0 + r % 7,
                              cols, ctx) for r in rows]


@pytest.mark.parametrize("cols", [2560, 6912])
def test_sweep_again_and_again(oracle, ctx, cols):
    import torch
    from lemonade_burn_b200 import ops
    lins = _linears(oracle, ctx, cols, [2560, 640, 640], cols)
    x = torch.randn(1, cols, generator=torch.Generator(device="cuda").manual_seed(cols), device="cuda")
    want = [w.view(-1) for w in ops.ternary_linear_multi(x.repeat(9, 1), lins)]  # the GEMM: the same integers and product of scales
    plan, outs = ops.Plan(ctx), [[torch.empty(l.rows, device="cuda") for l in lins] for _ in range(16)]
    for o in outs:
        plan.add(x, lins, o)
    plan.finalize()
    for _ in range(200):
        plan.run()
        for o in outs:
            for got, w in zip(o, want):
                assert torch.equal(got, w[:got.numel()])
    ctx.check_device_error()


@pytest.mark.parametrize("m", [1, 4, 8])
def test_few_rows_again_and_again(oracle, ctx, m):
    import torch
    from lemonade_burn_b200 import ops
    lins = _linears(oracle, ctx, 4096, [4096, 1024, 1024], 7)
    x = torch.randn(m, 4096, generator=torch.Generator(device="cuda").manual_seed(m), device="cuda")
    want = ops.ternary_linear_multi(x.repeat(9, 1), lins)
    for _ in range(500):
        for got, w in zip(ops.ternary_linear_multi(x, lins), want):
            assert torch.equal(got, w[:m])
    ctx.check_device_error()


@pytest.mark.parametrize("b", [1, 5])
def test_step_again_and_again(ctx, b):
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(2560, 6912, 20, 5, 4, 500, 1e-5, 500000.0, 300)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, b, "cuda"), ctx)
    c, toks = net.new_cache(b, 300), torch.arange(b, dtype=torch.int32, device="cuda")
    want = None
    for _ in range(500):
        c.pos.fill_(7)  # the row of the position is written again, with the same values
        c.host_len = 7
        got = net.forward(toks, c)
        want = got.clone() if want is None else want
        assert torch.equal(got, want)
    ctx.check_device_error()
