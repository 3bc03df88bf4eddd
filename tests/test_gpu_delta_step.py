"""The delta rule's decode step in both forms (everything asked for at once: four taps, heads and ranks of at most 128; and the general one) against the
prompt pass over the same tokens, which goes through other kernels. f32: the two differ by the order of sums alone; logits agree to 2e-4 of their
spread, the bound that the family's f32 tests hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VOCAB = 64


@pytest.mark.parametrize("heads,kv,dim,vdim,taps,low", [(2, 2, 128, 128, 4, 128), (4, 2, 64, 128, 4, 16), (2, 2, 128, 64, 4, 100), (3, 3, 40, 24, 4, 8), (2, 2, 128, 128, 3, 128),
                                                        (2, 2, 128, 128, 5, 16), (2, 2, 128, 128, 4, 160), (2, 2, 192, 64, 4, 16), (2, 1, 64, 160, 4, 16)])
def test_step_against_prompt(ctx, tmp_path, heads, kv, dim, vdim, taps, low):
    import torch
    from lemonade_burn_b200 import dugulorn
    cfg = dugulorn.make_config(VOCAB, 256, [dugulorn.delta_layer(heads, kv, dim, vdim, taps, 192)] * 2)
    dugulorn.save_checkpoint(tmp_path, cfg, dugulorn.random_checkpoint(cfg, dim + vdim + taps, low))
    net = dugulorn.NativeDugulorn(tmp_path, ctx, "float32")
    rng = np.random.default_rng(low)
    tokens = rng.integers(0, VOCAB, (3, 12)).astype(np.uint32)
    stepwise, whole = net.new_cache(3, 32), net.new_cache(1, 32)
    got = []
    for i in range(tokens.shape[1]):
        got.append(net.decode(torch.from_numpy(tokens[:, i].astype(np.int32)).cuda(), stepwise)[0].clone())
    got = torch.stack(got, 1).cpu().numpy()
    for s in range(3):
        net.reset_cache(whole)
        want = net.forward_rows(tokens[s], whole, list(range(tokens.shape[1])))
        assert np.abs(got[s] - want).max() <= 2e-4 * np.abs(want).max()
    ctx.check_device_error()


@pytest.mark.parametrize("heads,dim,vdim", [(20, 128, 128), (37, 64, 40), (149, 96, 24)])
def test_plain_step_of_many_blocks(ctx, heads, dim, vdim):
    """The plain rule's step holds the state in registers up to a block an SM and in shared memory beyond: sixteen sequences at once against the
    same sequences one by one. f32, the same products in sums of dim terms: at most dim roundings of sum |q S| apart, 2^-24 each."""
    import ctypes as C
    import torch
    from lemonade_burn_b200 import _lib, mixers
    lib, st, b = _lib.load(), torch.cuda.current_stream().cuda_stream, 16
    d = mixers.RecurrenceDesc(0, heads, heads, dim, vdim, 1)
    g = torch.Generator(device="cuda").manual_seed(heads)
    width = heads * (2 * dim + vdim)
    x = torch.randn(b, width, generator=g, device="cuda")
    floats = int(lib.lbk_recurrence_state_floats(C.byref(d)))
    pitch = floats // (heads * vdim)
    state = torch.zeros(b, heads, vdim, pitch, device="cuda")
    state[..., :dim] = torch.randn(b, heads, vdim, dim, generator=g, device="cuda")
    pos, active = torch.arange(b, dtype=torch.int32, device="cuda"), torch.ones(b, dtype=torch.int32, device="cuda")
    active[5] = 0
    decay, start = torch.rand(heads, generator=g, device="cuda"), state.clone()

    def run(rows, at, act, s, o):
        _lib.check(lib.lbk_recurrence(ctx.handle, 1, C.byref(d), rows.data_ptr(), width, rows.shape[0], -1, at.data_ptr(), act.data_ptr(), 64, decay.data_ptr(), None, None,
                                      None, None, None, None, s.data_ptr(), None, 0, o.data_ptr(), st))

    got, want, one = torch.empty(b, heads * vdim, device="cuda"), torch.empty(b, heads * vdim, device="cuda"), start.clone()
    run(x, pos, active, state, got)
    for i in range(b):
        run(x[i:i + 1], pos[i:i + 1], active[i:i + 1], one[i:i + 1], want[i:i + 1])
    bound = (dim + 8) * 2.0 ** -24 * (x.abs().max() ** 2 * dim * x.abs().max() + x.abs().max() * dim * start.abs().max())
    assert float((got - want).abs().max()) <= float(bound) and float(got.abs().max()) > 0
    assert torch.equal(state[5], start[5]) and not torch.equal(state[4], start[4])
    assert float((state - one).abs().max()) <= 4 * 2.0 ** -24 * float(state.abs().max())
    ctx.check_device_error()
