"""Weights that a kernel of this library writes right in front of the call that reads them. The kernels start beside the end of the one in front
(programmatic launches, each lets the next start at once), so a call that read its weights ahead would get what they were before: a head
of many rows keeps the writer waiting for some hundred microseconds, time enough for the reader to be there. Equality: the same call once all is settled."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


class Front:
    """Keeps the device busy: a launch whose end what follows on the stream has to wait for."""

    def __init__(self, ctx):
        import torch
        self.ctx, self.w = ctx, torch.zeros(160000, 2560, dtype=torch.bfloat16, device="cuda")
        self.x, self.out = torch.ones(1, 2560, device="cuda"), torch.empty(1, 160000, device="cuda")

    def launch(self, st):
        from lemonade_burn_b200 import _lib
        _lib.check(_lib.load().lbk_bf16_linear(self.ctx.handle, self.x.data_ptr(), 1, self.w.data_ptr(), 160000, 2560, self.out.data_ptr(), st))

    def vector(self, src, dst, st):
        """dst = src by a kernel: x += y on zeros."""
        from lemonade_burn_b200 import _lib
        _lib.check(_lib.load().lbk_add_inplace(self.ctx.handle, dst.data_ptr(), src.data_ptr(), src.numel(), st))


@pytest.fixture(scope="module")
def front(ctx):
    return Front(ctx)


@pytest.mark.parametrize("kv,cap", [(1, 1), (2, 64), (8, 512)])
def test_head_over_rows_just_appended(ctx, front, kv, cap):
    """lbk_bf16_linear of one row over cache rows that lbk_rope_kv_append writes."""
    import torch
    from lemonade_burn_b200 import _lib
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(kv + cap)
    table = torch.randn(kv * cap, 128, generator=g, device="cuda").to(torch.bfloat16)
    other = torch.zeros_like(table)
    q, k, v = (torch.randn(1, n * 128, generator=g, device="cuda") for n in (kv, kv, kv))
    cos, sin = torch.ones(cap, 128, device="cuda"), torch.zeros(cap, 128, device="cuda")
    pos, x = torch.tensor([cap - 1], dtype=torch.int32, device="cuda"), torch.randn(1, 128, generator=g, device="cuda")
    got, want = torch.empty(1, kv * cap, device="cuda"), torch.empty(1, kv * cap, device="cuda")
    head = lambda out: _lib.check(lib.lbk_bf16_linear(ctx.handle, x.data_ptr(), 1, table.data_ptr(), kv * cap, 128, out.data_ptr(), st))  # noqa: E731
    for _ in range(5):
        table[cap - 1::cap] = 0  # the rows that are appended
        torch.cuda.synchronize()
        front.launch(st)
        _lib.check(lib.lbk_rope_kv_append(ctx.handle, q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), 1, kv, kv, 128, cap,
                                          table.data_ptr(), other.data_ptr(), st))
        head(got)
        torch.cuda.synchronize()
        head(want)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and bool((want[0, cap - 1::cap] != 0).all())
    ctx.check_device_error()


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,n", [(1, 512), (3, 2560), (148, 8192)])
def test_norm_with_weights_just_written(ctx, front, rows, n, rms):
    import torch
    from lemonade_burn_b200 import _lib
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    x0, y, *src = (torch.randn(s, generator=g, device="cuda") for s in ((rows, n), (rows, n), (n,), (n,)))
    w, w_post = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")

    def norm():
        x, out = x0.clone(), torch.empty(rows, n, device="cuda")
        call = lib.lbk_sandwich_rms_norm if rms else lib.lbk_sandwich_norm
        return x, out, lambda: _lib.check(call(ctx.handle, x.data_ptr(), y.data_ptr(), w_post.data_ptr(), w.data_ptr(), rows, n, C.c_float(1e-6), out.data_ptr(), None, 0, st))

    for late, early in ((w, w_post), (w_post, w)):
        late.zero_()
        early.copy_(src[late is w])
        x, got, call = norm()
        torch.cuda.synchronize()
        front.launch(st)
        front.vector(src[late is w_post], late, st)
        call()
        torch.cuda.synchronize()
        xw, want, call = norm()
        call()
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(x, xw) and bool((got != 0).any())
    ctx.check_device_error()


@pytest.mark.parametrize("compute", [0, 1])
@pytest.mark.parametrize("rows", [1, 16])
def test_latents_with_weights_just_written(ctx, front, rows, compute):
    import torch
    from lemonade_burn_b200 import _lib, mixers
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    q_rank, kv_rank, rot, cap = 1536, 512, 64, 40
    f, m = mixers.rotation_frequencies(rot, 1e4, None)
    freq = torch.from_numpy(f).cuda()
    d = mixers.LatentDesc(4, 128, rot, 128, kv_rank, q_rank, freq.data_ptr(), m)
    g = torch.Generator(device="cuda").manual_seed(rows)
    z = torch.randn(rows, q_rank + kv_rank + rot, generator=g, device="cuda")
    pos, kind = torch.arange(rows, dtype=torch.int32, device="cuda"), torch.float32 if compute else torch.bfloat16
    src = torch.randn(q_rank, generator=g, device="cuda"), torch.randn(kv_rank, generator=g, device="cuda")
    w = torch.empty(q_rank, device="cuda"), torch.empty(kv_rank, device="cuda")

    def prep():
        cq, cache = torch.zeros(rows, q_rank, dtype=kind, device="cuda"), torch.zeros(rows, cap, lib.lbk_latent_pitch(C.byref(d)), dtype=kind, device="cuda")
        return cq, cache, lambda: _lib.check(lib.lbk_latent_prep(ctx.handle, compute, C.byref(d), z.data_ptr(), z.shape[1], rows, -1, pos.data_ptr(), cap, w[0].data_ptr(),
                                                                 w[1].data_ptr(), C.c_float(1e-6), cq.data_ptr(), q_rank, cache.data_ptr(), st))

    for late in (0, 1):
        w[late].zero_()
        w[1 - late].copy_(src[1 - late])
        cq, cache, call = prep()
        torch.cuda.synchronize()
        front.launch(st)
        front.vector(src[late], w[late], st)
        call()
        torch.cuda.synchronize()
        cqw, want, call = prep()
        call()
        torch.cuda.synchronize()
        assert torch.equal(cq, cqw) and torch.equal(cache, want) and bool((cq != 0).any())
    ctx.check_device_error()
