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


class Device:
    """An allocation of its own of so many bytes (512 lie behind any: nothing else is there to be hit)."""

    def __init__(self, size, managed=False):
        self.lib, self.at = C.CDLL("libcuda.so.1"), C.c_uint64()
        status = self.lib.cuMemAllocManaged(C.byref(self.at), C.c_size_t(size), C.c_uint(1)) if managed else self.lib.cuMemAlloc_v2(C.byref(self.at), C.c_size_t(size))
        assert status == 0
        self.size = size

    def tensor(self, dtype, n, offset=0):
        import torch
        raw = torch.empty(n * 4, dtype=torch.uint8, device="cuda")
        assert self.lib.cuMemcpyDtoD_v2(C.c_uint64(raw.data_ptr()), C.c_uint64(self.at.value + offset), C.c_size_t(n * 4)) == 0
        return raw.view(dtype)

    def free(self):
        self.lib.cuMemFree_v2(self.at)


def _decode(net, cache, tokens, logits, nxt):
    import torch
    from lemonade_burn_b200 import _lib
    return _lib.load().lbk_model_decode(net.handle, cache, C.c_void_p(tokens), C.c_void_p(logits), C.c_void_p(nxt), C.c_void_p(torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("b", [1, 5])
def test_memory_of_other_kinds(ctx, tmp_path, b):
    """Results and tokens in managed memory, and in allocations that end with them."""
    import torch
    net, vocab = _net(ctx, tmp_path, 100), 100
    toks = torch.arange(b, dtype=torch.int32, device="cuda")
    want, nxt = torch.zeros(b, vocab, device="cuda"), torch.zeros(b, dtype=torch.int32, device="cuda")
    assert _decode(net, net.new_cache(b, 8), toks.data_ptr(), want.data_ptr(), nxt.data_ptr()) == 0
    for managed in (True, False):
        t, l, n = Device(b * 4, managed), Device(b * vocab * 4, managed), Device(b * 4, managed)
        assert t.lib.cuMemcpyDtoD_v2(t.at, C.c_uint64(toks.data_ptr()), C.c_size_t(b * 4)) == 0
        torch.cuda.synchronize()
        assert _decode(net, net.new_cache(b, 8), t.at.value, l.at.value, n.at.value) == 0
        torch.cuda.synchronize()
        assert torch.equal(l.tensor(torch.float32, b * vocab).view(b, vocab), want) and torch.equal(n.tensor(torch.int32, b), nxt)
        for d in (t, l, n):
            d.free()
    ctx.check_device_error()


def test_memory_that_does_not_hold_the_call_is_refused(ctx, tmp_path):
    """By a status, as a copy refuses it; and a step that was refused for its tokens leaves nothing behind for the next one to write to."""
    import torch
    net, vocab = _net(ctx, tmp_path, 100), 100
    toks = torch.zeros(1, dtype=torch.int32, device="cuda")
    small, few = Device(vocab * 4 - 256), Device(4)
    assert _decode(net, net.new_cache(1, 8), toks.data_ptr(), small.at.value, None) != 0
    logits, cache = torch.zeros(5, vocab, device="cuda"), net.new_cache(5, 8)
    assert _decode(net, cache, few.at.value, logits.data_ptr(), None) != 0
    good = torch.zeros(5, dtype=torch.int32, device="cuda")
    assert _decode(net, cache, good.data_ptr(), None, None) == 0
    torch.cuda.synchronize()
    assert not bool(logits.any())
    small.free()
    few.free()
    ctx.check_device_error()


def _greedy(row):
    """sample.rs:17-25: the first index whose value is above all in front of it; comparisons with a NaN do not hold."""
    best, at = row[0], 0
    for i, v in enumerate(row):
        if v > best:
            best, at = v, i
    return at


@pytest.mark.parametrize("vocab", [257, 5003])
def test_greedy_token_of_unusual_rows(ctx, tmp_path, vocab):
    """A NaN in front, NaNs inside, rows of -inf but for one, equal maxima in two parts of a row, the maximum at either end."""
    import torch
    from lemonade_burn_b200 import _lib, dugulorn
    cfg, token = dugulorn.make_config(vocab, 256, [dugulorn.delta_layer(2, 2, 64, 64, 4, 192)]), 7
    tensors = dugulorn.random_checkpoint(cfg, 5, 16)
    name = next(k for k, v in tensors.items() if v.shape == (vocab, 256))
    table = torch.from_numpy(tensors[name].view(np.int16)).view(torch.bfloat16)

    def step(change):
        t = table.clone()
        change(t)
        folder = tmp_path / f"m{step.count}"
        step.count += 1
        folder.mkdir()
        dugulorn.save_checkpoint(folder, cfg, {**tensors, name: t.view(torch.int16).numpy().view(np.uint16)})
        net = dugulorn.NativeDugulorn(folder, ctx, "float32")
        logits, nxt = torch.zeros(2, vocab, device="cuda"), torch.full((2,), -1, dtype=torch.int32, device="cuda")
        toks = torch.tensor([token, token], dtype=torch.int32, device="cuda")
        assert _decode(net, net.new_cache(2, 8), toks.data_ptr(), logits.data_ptr(), nxt.data_ptr()) == 0
        argmax = torch.empty_like(nxt)
        _lib.check(_lib.load().lbk_argmax(ctx.handle, logits.data_ptr(), 2, vocab, argmax.data_ptr(), torch.cuda.current_stream().cuda_stream))
        rows = logits.cpu().numpy()
        assert nxt.tolist() == [_greedy(r) for r in rows] and torch.equal(nxt, argmax)
        return rows[0], int(nxt[0])

    step.count = 0
    plain, top = step(lambda t: None)
    assert top == int(plain.argmax())
    along = torch.sign(torch.from_numpy(plain[top:top + 1])) * table[top].float()  # a row whose logit is positive

    def rows_are(places, value):
        def change(t):
            for i in places:
                t[i] = value
        return change

    assert step(rows_are([0], float("nan")))[1] == 0
    row, at = step(rows_are([9, 64, vocab - 1], float("nan")))
    assert np.isnan(row[[9, 64, vocab - 1]]).all() and at == int(np.nanargmax(row))
    for places in ([100, vocab - 3], [0, vocab - 1], [vocab - 1], [79, 80]):
        row, at = step(rows_are(places, (along * 64).to(torch.bfloat16)))
        assert at == places[0] and (row[places] == row[at]).all()
    low = torch.zeros(256)
    low[int(along.abs().argmax())] = -torch.sign(along[int(along.abs().argmax())]) * float("inf")
    others = [i for i in range(vocab) if i != token]
    row, at = step(rows_are(others, low.to(torch.bfloat16)))
    if not np.isnan(row).any():
        assert at == (token if row[others[0]] == -np.inf else 0)
    ctx.check_device_error()
