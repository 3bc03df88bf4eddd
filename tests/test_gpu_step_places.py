"""The decode step in one launch with one sequence: what one part hands to the next lies in two places that the layers take in turn, through all
launches. Layer counts that leave the turn even and odd, one slice of the positions, few and many, blocks without tiles: step after step against
the step with a kernel per operation. The bar between the two routes is 2e-3 of the largest logit; a row with a code on a rounding boundary may come
out further apart, 0.02 at most (test_gpu_step.py has the bound), and not most of them. And a position past the cache, which has no values to hand on, ends the launch and leaves the next one sound."""
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-3


@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("hidden,inner,heads,kv,cap", [(512, 768, 4, 1, 40), (512, 1100, 4, 4, 130), (1280, 3408, 10, 5, 300), (2560, 6912, 20, 5, 2100)])
def test_turns(ctx, hidden, inner, heads, kv, cap, layers):
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(hidden, inner, heads, kv, layers, 500, 1e-5, 500000.0, cap)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, hidden + layers, "cuda"), ctx)
    assert net._step.supported(1, cap)
    one, ref = net.new_cache(1, cap), net.new_cache(1, cap)
    g = torch.Generator(device="cuda").manual_seed(layers)
    for a, r in ((one.k, ref.k), (one.v, ref.v)):
        a.copy_(torch.randn(a.shape, generator=g, device="cuda"))
        r.copy_(a)
    for c in (one, ref):
        c.pos.fill_(cap - 7)
        c.host_len = cap - 7
    apart = 0
    for i in range(7):
        toks = torch.randint(0, 500, (1,), dtype=torch.int32, generator=g, device="cuda")
        got, want = net.forward(toks, one), net.forward(toks, ref, splits=model.attention_splits(cap))
        err = float((got - want).abs().max() / want.abs().max())
        assert err <= 0.02, (i, err)
        apart += err > TOL
    assert apart <= 3
    ctx.check_device_error()


def test_position_past_the_cache(ctx):
    import torch
    from lemonade_burn_b200 import _lib, model
    for cap in (16, 300):  # one slice, several
        cfg = model.Config(512, 768, 4, 1, 3, 500, 1e-5, 500000.0, cap)
        net = model.BitNet(cfg, model.random_checkpoint(cfg, cap), ctx)
        c, toks = net.new_cache(1, cap), torch.tensor([7], dtype=torch.int32, device="cuda")
        want = net.forward(toks, c).clone()
        c.pos.fill_(cap)
        net.forward(toks, c)
        with pytest.raises(_lib.LbkError) as e:
            ctx.check_device_error()
        assert e.value.status != 5  # no wait ran out
        c.pos.zero_()
        c.host_len = 0
        assert torch.equal(net.forward(toks, c), want)
        ctx.check_device_error()
