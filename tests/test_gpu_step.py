"""The decode step in one launch (lbk_step_*) against the step with a kernel per operation, which the decoder tests hold to the
oracle: same integers in the projections, float sums in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-3  # of max |logit|: the decoder tests' bar between routes


@pytest.mark.parametrize("b", [1, 2, 8, 9, 16])
@pytest.mark.parametrize("hidden,inner,heads,kv,start,cap", [
    (512, 768, 4, 1, 0, 40),        # fewer tiles than SMs, one slice, from an empty cache
    (512, 1100, 4, 4, 61, 70),      # rows and columns that end inside a tile and a block, one query head per KV head
    (1280, 3408, 10, 5, 127, 300),  # two query heads per KV head, a slice boundary at the new position
    (2560, 6912, 20, 5, 900, 1024),
])
def test_one_launch_matches_a_kernel_per_operation(ctx, hidden, inner, heads, kv, start, cap, b):
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(hidden, inner, heads, kv, 2, 1000, 1e-5, 500000.0, cap)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, hidden + b), ctx)
    one, ref = net.new_cache(b, cap), net.new_cache(b, cap)
    assert net._step.supported(b, cap)
    g = torch.Generator(device="cuda").manual_seed(b)
    for a, r in ((one.k, ref.k), (one.v, ref.v)):
        a.copy_(torch.randn(a.shape, generator=g, device="cuda"))
        r.copy_(a)
    for c in (one, ref):
        c.pos.fill_(start)
        c.host_len = start
    steps = min(4, cap - start)
    for _ in range(steps):
        toks = torch.randint(0, 1000, (b,), dtype=torch.int32, generator=g, device="cuda")
        got, want = net.forward(toks, one), net.forward(toks, ref, splits=model.attention_splits(cap))
        assert (got - want).abs().max() <= TOL * want.abs().max()
    assert one.len == ref.len == start + steps
    new = slice(start, start + steps)
    for a, r in ((one.k, ref.k), (one.v, ref.v)):
        assert torch.equal(a[:, :, :, :start], r[:, :, :, :start]) and torch.equal(a[:, :, :, start + steps:], r[:, :, :, start + steps:])
        # values on either side of a rounding boundary of the cache's bf16 lie one of its steps apart: 2^-7 of the value at most
        assert (a[:, :, :, new].float() - r[:, :, :, new].float()).abs().max() <= (2 * TOL + 2 ** -7) * r[:, :, :, new].float().abs().max()
    ctx.check_device_error()


def test_step_past_the_cache_reports_and_leaves_the_cache(ctx):
    import torch
    from lemonade_burn_b200 import _lib, model
    cfg = model.Config(512, 768, 4, 1, 1, 1000, 1e-5, 500000.0, 16)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 3), ctx)
    c = net.new_cache(2, 16)
    c.pos.fill_(16)  # the device-side position alone: what a replayed step would meet
    net.forward(torch.tensor([1, 2], dtype=torch.int32, device="cuda"), c)
    with pytest.raises(_lib.LbkError):
        ctx.check_device_error()
    assert int(c.k.abs().sum()) == 0 and int(c.v.abs().sum()) == 0
    c.pos.zero_()
    c.host_len = 0
    out = net.forward(torch.tensor([1, 2], dtype=torch.int32, device="cuda"), c)  # and the next launch is a good one
    ctx.check_device_error()
    assert np.isfinite(out.cpu().numpy()).all()
