"""What a recorded step hands out: logits and greedy tokens in the caller's memory, wanted or not, aligned or not, on the device or in pinned host memory;
vocabularies of fewer columns than parts, of whole 16-byte units and not; and a step without a caller behind one with. Equality: the same values are
copied, and the greedy token is the first of the largest (a row that is all alike: column 0)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(ctx, path, vocab):
    from lemonade_burn_b200 import dugulorn
    cfg = dugulorn.make_config(vocab, 256, [dugulorn.delta_layer(2, 2, 64, 64, 4, 192)])
    dugulorn.save_checkpoint(path, cfg, dugulorn.random_checkpoint(cfg, 5, 16))
    return dugulorn.NativeDugulorn(path, ctx, "float32")


@pytest.mark.parametrize("vocab", [3, 64, 255, 257, 1000, 5003])
@pytest.mark.parametrize("b", [1, 3, 16])
def test_results_reach_the_caller(ctx, tmp_path, vocab, b):
    import torch
    from lemonade_burn_b200 import _lib
    lib, net = _lib.load(), _net(ctx, tmp_path, vocab)
    toks = torch.arange(b, dtype=torch.int32, device="cuda") % vocab
    stream = torch.cuda.current_stream().cuda_stream

    def step(logits, nxt, tokens=toks):
        cache = net.new_cache(b, 8)
        _lib.check(lib.lbk_model_decode(net.handle, cache, C.c_void_p(tokens.data_ptr()), C.c_void_p(logits.data_ptr() if logits is not None else None),
                                        C.c_void_p(nxt.data_ptr() if nxt is not None else None), C.c_void_p(stream)))
        torch.cuda.synchronize()
        return cache

    want, nxt = torch.zeros(b, vocab, device="cuda"), torch.full((b,), -1, dtype=torch.int32, device="cuda")
    step(want, nxt)
    assert torch.isfinite(want).all() and float(want.abs().max()) > 0
    assert np.array_equal(nxt.cpu().numpy(), want.cpu().numpy().argmax(1))
    shifted, nxt2 = torch.zeros(b * vocab + 1, device="cuda"), torch.zeros_like(nxt)  # four bytes past a 16-byte boundary
    step(shifted[1:], nxt2)
    assert torch.equal(shifted[1:].view(b, vocab), want) and float(shifted[0]) == 0 and torch.equal(nxt2, nxt)
    only, none = torch.zeros_like(want), torch.zeros_like(nxt)
    step(only, None)
    step(None, none)
    assert torch.equal(only, want) and torch.equal(none, nxt)
    host, hnxt = torch.zeros(b, vocab).pin_memory(), torch.zeros(b, dtype=torch.int32).pin_memory()
    step(host, hnxt, toks.cpu().pin_memory())
    assert torch.equal(host, want.cpu()) and torch.equal(hnxt, nxt.cpu())
    # a step of the library's own behind a caller's leaves the caller's memory alone
    kept, keptn = torch.zeros_like(want), torch.zeros_like(nxt)
    cache = step(kept, keptn)
    if b == 1:
        before = kept.clone()
        net.forward(np.array([2 % vocab], np.uint32), cache)
        assert torch.equal(kept, before)
    ctx.check_device_error()
