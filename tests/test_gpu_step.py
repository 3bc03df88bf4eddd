"""The decode step in one launch (lbk_step_*) against the step with a kernel per operation (`splits` given), which the decoder tests hold to
the oracle by name. From equal rows the projections' sums are the same integers but for codes on a rounding boundary: the one rounds
y (127 / max |y|) with y = x w, the other (x r w) (127 / max |x r w|). Float sums come in another order."""
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
    from lemonade_burn_b200 import model
    cfg = model.Config(hidden, inner, heads, kv, 2, 1000, 1e-5, 500000.0, cap)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, hidden + b), ctx)
    assert net._step.supported(b, cap)
    _compare(ctx, net, b, start, cap, TOL)


@pytest.mark.parametrize("hidden,inner,heads,kv,most", [
    (4096, 14336, 32, 8, 10),   # eight float4 of the feed-forward row a thread; two stages a ring at nine and ten sequences
    (5120, 7168, 40, 10, 16),   # four and four
    (8192, 16384, 64, 16, 9),   # four and eight: the longest rows that are served
])
def test_wide_models(ctx, hidden, inner, heads, kv, most):
    """A row whose codes fall on the two sides of a rounding boundary in the two routes comes out apart: one turned code of about 35 changes a
    product of k = 4096 terms by r = 1 / (35 sqrt(k)) = 0.00045 of itself; that moves the next quantiser's codes by 35 r and turns that share of
    them, a change of sqrt(r / 35): 0.0036, 0.010 and 0.017 behind the three quantisers that follow. With 26000 to 41000 codes a row, each turned
    with a chance of 4e-6 to 3e-5, that meets a row in ten at least; the others keep the bar."""
    from lemonade_burn_b200 import model
    cap = 80
    cfg = model.Config(hidden, inner, heads, kv, 1, 1000, 1e-5, 500000.0, cap)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, hidden, "cuda"), ctx)
    assert [b for b in range(1, 18) if net._step.supported(b, cap)] == list(range(1, most + 1))  # more rows do not fit in shared memory
    apart = [r for b in sorted({1, 3, 8, 9, most}) for r in _compare(ctx, net, b, 61, cap, 0.02)]
    assert sum(apart) <= len(apart) // 2, apart


def _compare(ctx, net, b, start, cap, tol):
    """Steps by both routes; which rows of theirs were further apart than TOL, none further than `tol`."""
    import torch
    from lemonade_burn_b200 import model
    one, ref = net.new_cache(b, cap), net.new_cache(b, cap)
    g = torch.Generator(device="cuda").manual_seed(b)
    for a, r in ((one.k, ref.k), (one.v, ref.v)):
        a.copy_(torch.randn(a.shape, generator=g, device="cuda"))
        r.copy_(a)
    for c in (one, ref):
        c.pos.fill_(start)
        c.host_len = start
    steps, apart = min(4, cap - start), []
    for _ in range(steps):
        toks = torch.randint(0, 1000, (b,), dtype=torch.int32, generator=g, device="cuda")
        got, want = net.forward(toks, one), net.forward(toks, ref, splits=model.attention_splits(cap))
        err = (got - want).abs().amax(1) / want.abs().max()
        assert err.max() <= tol, err
        apart += (err > TOL).tolist()
    assert one.len == ref.len == start + steps
    new = slice(start, start + steps)
    for a, r in ((one.k, ref.k), (one.v, ref.v)):
        assert torch.equal(a[:, :, :, :start], r[:, :, :, :start]) and torch.equal(a[:, :, :, start + steps:], r[:, :, :, start + steps:])
        # values on either side of a rounding boundary of the cache's bf16 lie one of its steps apart: 2^-7 of the value at most
        assert (a[:, :, :, new].float() - r[:, :, :, new].float()).abs().max() <= (2 * TOL + 2 ** -7) * r[:, :, :, new].float().abs().max()
    ctx.check_device_error()
    return apart


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


def test_steps_of_two_sizes_from_two_threads(ctx):
    """Two models whose steps take the same kernel with unequal shared memory, each launched from a thread and on a stream of its own, with
    nothing but the call in the loop: no launch fails, and both give what they give alone."""
    import threading
    import torch
    from lemonade_burn_b200 import _lib, model
    lib, cap, failed, jobs = _lib.load(), 64, [], []
    for hidden, inner, heads, kv in ((512, 768, 4, 1), (1280, 3408, 10, 5)):
        cfg = model.Config(hidden, inner, heads, kv, 1, 500, 1e-5, 500000.0, cap)
        net = model.BitNet(cfg, model.random_checkpoint(cfg, hidden), ctx)
        c, x, out, h = net.new_cache(1, cap), torch.randn(1, hidden, device="cuda"), torch.zeros(2, hidden, device="cuda"), net._step.handle
        work = torch.zeros(int(lib.lbk_step_work_bytes(h, 1, cap)), dtype=torch.uint8, device="cuda")
        ptrs = [t.data_ptr() for t in (x, c.k, c.v)], [t.data_ptr() for t in (net.cos, net.sin, c.pos)]
        jobs.append((net, c, x, work, out, torch.cuda.Stream(), lambda row, stream, h=h, a=ptrs, e=c.k.stride(0), w=work, o=out:
                     lib.lbk_step_run(h, 1, cap, *a[0], e, *a[1], 0, w.data_ptr(), o[row].data_ptr(), stream)))
        _lib.check(jobs[-1][-1](0, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()

    def steps(stream, call):
        for _ in range(4000):
            if call(1, stream) != 0:
                failed.append(lib.lbk_last_error())
                return

    threads = [threading.Thread(target=steps, args=(j[5].cuda_stream, j[6])) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    for j in jobs:
        assert torch.equal(j[4][0], j[4][1])
    ctx.check_device_error()


def test_stream_with_a_part_of_the_device(ctx, tmp_path):
    """On a stream whose green context has some of the SMs the step cannot be resident as a whole: the models decode all the same, and the
    refused launch leaves no error behind for the next call."""
    import torch
    from lemonade_burn_b200 import _lib, model
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("no green contexts")
    cfg = model.Config(512, 768, 4, 1, 2, 1000, 1e-5, 500000.0, 64)
    tensors = model.random_checkpoint(cfg, 3)
    model.save_checkpoint(tmp_path, cfg, tensors)
    net, nat = model.BitNet(cfg, tensors, ctx), model.NativeBitNet(tmp_path, ctx)
    toks = torch.tensor([1, 2], dtype=torch.int32, device="cuda")
    chain = net.forward(toks, net.new_cache(2, 64), splits=model.attention_splits(64))
    step = net.forward(toks, net.new_cache(2, 64))
    work = torch.zeros(int(_lib.load().lbk_step_work_bytes(net._step.handle, 2, 64)), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    part = green_contexts.GreenContext.create(32, 0)
    with torch.cuda.stream(part.Stream()):
        assert not net._step.supported(2, 64)
        got, native = net.forward(toks, net.new_cache(2, 64)), nat.decode(toks, nat.new_cache(2, 64))[0]
        c, x = net.new_cache(2, 64), torch.zeros(2, 512, device="cuda")
        args = [t.data_ptr() for t in (x, c.k, c.v)], [t.data_ptr() for t in (net.cos, net.sin, c.pos)]
        status = _lib.load().lbk_step_run(net._step.handle, 2, 64, *args[0], c.k.stride(0), *args[1], 0, work.data_ptr(), x.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream)
        assert status != 0 and b"multiprocessors" in _lib.load().lbk_last_error()
        again = net.forward(toks, net.new_cache(2, 64))
    torch.cuda.synchronize()
    assert torch.equal(got, chain) and torch.equal(again, chain) and torch.equal(native, step)
    assert net._step.supported(2, 64)
    ctx.check_device_error()
    nat.close()


def test_caches_of_one_shape_step_on_two_streams(ctx):
    """Each cache has a work buffer of its own, which goes with it: the launches of two caches count their arrivals apart."""
    import weakref
    import torch
    from lemonade_burn_b200 import model
    cap, b = 48, 2
    cfg = model.Config(1280, 3408, 10, 5, 2, 500, 1e-5, 500000.0, cap)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 9), ctx)
    a, c = net.new_cache(b, cap), net.new_cache(b, cap)
    assert a.step_work.data_ptr() != c.step_work.data_ptr()
    gone = weakref.ref(c.step_work)
    del c
    assert gone() is None
    runs = []
    for i in range(2):
        g = torch.Generator(device="cuda").manual_seed(i)
        cache, x, out = net.new_cache(b, cap), torch.randn(b, 1280, generator=g, device="cuda"), torch.zeros(cap, b, 1280, device="cuda")
        runs.append((cache, x, out, torch.cuda.Stream()))
    pos = torch.arange(cap, dtype=torch.int32, device="cuda")

    def step(run, t):
        cache, x, out, _ = run
        net._step.run(x, cache.k, cache.v, net.cos, net.sin, pos[t:], 0, out[t], cache.step_work)

    want = []
    for run in runs:  # one after the other
        for t in range(cap):
            step(run, t)
        want.append(run[2].clone())
        run[0].k.zero_()
        run[0].v.zero_()
        run[2].zero_()
    torch.cuda.synchronize()
    for t in range(cap):  # in turn, nothing between the streams
        for run in runs:
            with torch.cuda.stream(run[3]):
                step(run, t)
    torch.cuda.synchronize()
    assert all(torch.equal(run[2], w) for run, w in zip(runs, want))
    ctx.check_device_error()


def test_models_that_the_step_does_not_take(ctx):
    """No layers, heads of another size, query heads that KV heads do not divide, a projection of other rows: such models are made as before, and
    the one without layers runs."""
    import torch
    from lemonade_burn_b200 import model
    for hidden, heads, kv, layers in ((256, 2, 1, 0), (256, 4, 2, 1), (384, 3, 2, 1)):
        cfg = model.Config(hidden, 256, heads, kv, layers, 300, 1e-5, 500000.0, 16)
        net = model.BitNet(cfg, model.random_checkpoint(cfg, 1), ctx)
        assert net._step is None
        if not layers:
            toks = torch.tensor([3, 4], dtype=torch.int32, device="cuda")
            x = net.lm_head[toks.long()].double()
            want = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * net.final_norm.double() @ net.lm_head.double().T
            got = net.forward(toks, net.new_cache(2, 16))
            assert (got - want).abs().max() <= TOL * want.abs().max()
    cfg = model.Config(256, 256, 2, 1, 1, 300, 1e-5, 500000.0, 16)
    tensors = model.random_checkpoint(cfg, 1)
    tensors["model.layers.0.self_attn.v_proj.qweight"] = tensors["model.layers.0.self_attn.v_proj.qweight"].repeat(2, 1)
    assert model.BitNet(cfg, tensors, ctx)._step is None
    ctx.check_device_error()


def test_step_follows_weights_that_are_put_in_later(ctx):
    """`layers` and `final_norm` are read at every call: another projection, another norm, a norm's storage exchanged under it."""
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(512, 768, 4, 1, 2, 500, 1e-5, 500000.0, 24)
    net, other = (model.BitNet(cfg, model.random_checkpoint(cfg, s), ctx) for s in (1, 2))
    toks = torch.tensor([3, 4], dtype=torch.int32, device="cuda")
    forward = lambda **kw: net.forward(toks, net.new_cache(2, 24), **kw)  # noqa: E731
    old, kept = [forward()], []  # what is taken out stays alive, so that a step that missed the change reads old weights and not free memory

    def check():
        got, want = forward(), forward(splits=model.attention_splits(24))
        assert (got - want).abs().max() <= TOL * want.abs().max()
        assert (got - old[0]).abs().max() > 10 * TOL * want.abs().max()
        old[0] = got

    for layer, name in ((0, "gate"), (1, "attn_sub_norm")):
        kept.append(net.layers[layer][name])
        net.layers[layer][name] = other.layers[layer][name] if name == "gate" else 3.0 * kept[-1].flip(0)
        check()
    kept.append(net.final_norm)
    net.final_norm = 2.0 * net.final_norm.flip(0)
    check()
    kept.append(net.layers[0]["ffn_sub_norm"].data)
    net.layers[0]["ffn_sub_norm"].data = torch.linspace(-2.0, 2.0, 768, device="cuda")
    check()
    ctx.check_device_error()


@pytest.mark.parametrize("b", [1, 3])
def test_step_whose_waits_run_out(ctx, b):
    """A count that nothing ever reaches: with a short limit every wait gives up, the launch ends, the status says so, and with the counts
    made zeros again the same buffers give the right rows."""
    import torch
    from lemonade_burn_b200 import _lib, model
    lib = _lib.load()
    cfg = model.Config(512, 768, 4, 1, 2, 500, 1e-5, 500000.0, 300)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 4), ctx)
    c, toks = net.new_cache(b, 300), torch.arange(b, dtype=torch.int32, device="cuda")
    want = net.forward(toks, c)
    ctx.check_device_error()
    assert lib.lbk_step_set_wait_limit(net._step.handle, 0) != 0
    _lib.check(lib.lbk_step_set_wait_limit(net._step.handle, 2000))
    c.step_work.zero_()
    c.step_work.view(torch.int32)[0] = 1  # one barrier that no block has come to
    c.pos.zero_()
    net.forward(toks, c)
    with pytest.raises(_lib.LbkError) as e:
        ctx.check_device_error()
    assert e.value.status == 5
    c.step_work.zero_()
    _lib.check(lib.lbk_step_set_wait_limit(net._step.handle, 1 << 20))
    c.pos.zero_()
    assert torch.equal(net.forward(toks, c), want)
    ctx.check_device_error()


def test_step_is_freed_after_its_context():
    """As a weight that borrows its memory can be: nothing of the context is looked at."""
    import torch
    from lemonade_burn_b200 import model, ternary
    own = ternary.Context(0)
    cfg = model.Config(512, 768, 4, 1, 1, 500, 1e-5, 500000.0, 24)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 1), own)
    net.forward(torch.tensor([3], dtype=torch.int32, device="cuda"), net.new_cache(1, 24))
    own.check_device_error()
    step, net._step = net._step, None
    own.close()
    assert step.ctx._lib.lbk_step_free(step.handle) == 0
    step.handle = None


def test_step_of_more_layers_than_memory_is_refused(ctx):
    """A status, and no C++ exception through the C entry."""
    import ctypes as C
    from lemonade_burn_b200 import _lib
    out, one = C.c_void_p(), (C.c_void_p * 1)()
    status = _lib.load().lbk_step_create(ctx.handle, 1 << 58, one, one, C.c_void_p(16), 4, 1, C.c_float(1e-5), C.byref(out))
    assert status == 6 and not out.value


def test_codes_on_a_rounding_boundary(ctx):
    """From equal rows the step's codes differ from those of the norm and quantise kernels by one where y (127 / max |y|) and (x r w) (127 / max |x r w|)
    lie on two sides of a half. Both are four roundings away from the exact value at most, 127 * 4 * 2^-24 = 3e-5 of a code: at most one code in
    16000 or so on each side, 0.16 of the rows of 2560. Seen in the query rows that a step of one layer leaves in its work buffer."""
    import torch
    from lemonade_burn_b200 import _lib, model, ops
    lib, b, rows, turned = _lib.load(), 16, 0, 0
    cfg = model.Config(2560, 6912, 20, 5, 1, 1000, 1e-5, 500000.0, 8)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 12, "cuda"), ctx)
    c, l = net.new_cache(b, 8), net.layers[0]
    for i in range(20):
        toks = torch.randint(0, 1000, (b,), dtype=torch.int32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i))
        c.pos.zero_()
        c.host_len = 0
        net.forward(toks, c)
        got = c.step_work[768:768 + b * 2560 * 4].view(torch.float32).view(b, 2560)  # behind three counters' places of 256 bytes
        x = net.lm_head[toks.long()].float()
        n = torch.empty_like(x)
        _lib.check(lib.lbk_rms_norm(ctx.handle, x.data_ptr(), l["input_norm"].data_ptr(), b, 2560, 1e-5, n.data_ptr(), torch.cuda.current_stream().cuda_stream))
        want = ops.ternary_linear(n, l["q"])
        units = (got - want) * (127.0 / n.abs().amax(1, keepdim=True)) * l["q"].scale  # of the projection's whole sums
        assert (units - units.round()).abs().max() < 0.01 and units.abs().max() < 8
        rows += b
        turned += int((units.abs() > 0.5).any(1).sum())
    assert turned <= 0.16 * rows, (turned, rows)
    ctx.check_device_error()


def test_cache_of_fewer_layers_is_refused(ctx):
    """By both routes; and a model that has lost its layers still runs."""
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(512, 768, 4, 1, 2, 500, 1e-5, 500000.0, 24)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 1), ctx)
    short = model.Config(512, 768, 4, 1, 1, 500, 1e-5, 500000.0, 24)
    tok = torch.tensor([3], dtype=torch.int32, device="cuda")
    for kw in ({}, {"splits": 1}):
        with pytest.raises(IndexError):
            net.forward(tok, model.KvCache(short, 1, 24, "cuda"), **kw)
    net.layers = net.layers[:1]
    got, want = net.forward(tok, net.new_cache(1, 24)), net.forward(tok, net.new_cache(1, 24), splits=1)
    assert (got - want).abs().max() <= TOL * want.abs().max()
    net.layers = []
    assert torch.equal(net.forward(tok, net.new_cache(1, 24)), net.forward(tok, net.new_cache(1, 24), splits=1))
    ctx.check_device_error()


def test_captured_step_survives_other_weights(ctx):
    """A graph that a program has captured goes on with the weights that it was captured with, also after the model has been given
    others and has stepped with them on the same cache."""
    import torch
    from lemonade_burn_b200 import model
    cfg = model.Config(512, 768, 4, 1, 2, 500, 1e-5, 500000.0, 24)
    net = model.BitNet(cfg, model.random_checkpoint(cfg, 1), ctx)
    c, tok = net.new_cache(1, 24), torch.tensor([3], dtype=torch.int32, device="cuda")
    net.forward(tok, c)
    net.forward(tok, net.new_cache(1, 24), splits=model.attention_splits(24))  # its buffers are there before anything is captured
    torch.cuda.synchronize()
    graph, kept = torch.cuda.CUDAGraph(), net.layers[0]["gate"]
    with torch.cuda.graph(graph):
        out = net.forward(tok, c)

    def at_start(call):
        c.pos.zero_()
        c.host_len = 0
        call()

    at_start(graph.replay)
    want = out.clone()
    net.layers[0]["gate"] = net.layers[1]["gate"]
    got = []
    at_start(lambda: got.append(net.forward(tok, c)))
    assert len(net._old_steps) == 1 and not torch.equal(got[0], want)
    junk = [torch.full((4096,), 255, dtype=torch.uint8, device="cuda") for _ in range(200)]  # what was given back is used again
    at_start(graph.replay)
    assert torch.equal(out, want) and kept is not net.layers[0]["gate"] and junk
    with torch.cuda.graph(torch.cuda.CUDAGraph()):  # other weights during a capture: a kernel per operation
        net.layers[0]["gate"] = kept
        at_start(lambda: net.forward(tok, c))
    ctx.check_device_error()
