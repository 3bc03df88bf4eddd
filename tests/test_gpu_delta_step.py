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
