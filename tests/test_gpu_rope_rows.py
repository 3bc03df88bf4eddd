"""lbk_rope_kv_append_rows: a row's bits do not depend on where its buffers lie or how many rows go with it."""
import pytest

pytestmark = pytest.mark.gpu


def _place(values, shift):
    """A copy of `values` that starts `shift` elements behind a 16-byte boundary."""
    import torch
    room = torch.empty(values.numel() + 8, dtype=values.dtype, device="cuda")
    at = room[shift:shift + values.numel()].view(values.shape)
    at.copy_(values)
    return at


@pytest.mark.parametrize("hd", [128, 64, 8, 12])  # 12: halves of six values, which no form takes four at a time
@pytest.mark.parametrize("n,nh,kvh", [(1, 4, 1), (33, 5, 5), (300, 20, 5)])
def test_rope_rows_whatever_the_alignment(ctx, hd, n, nh, kvh):
    import torch
    from lemonade_burn_b200 import _lib
    lib, st, pos0, cap, seq = _lib.load(), torch.cuda.current_stream().cuda_stream, 3, n + 5, 1
    g = torch.Generator(device="cuda").manual_seed(hd + n)
    q, k, v, cos, sin = (torch.randn(s, generator=g, device="cuda") for s in ((n, nh, hd), (n, kvh, hd), (n, kvh, hd), (cap, hd), (cap, hd)))
    pos = torch.tensor([pos0], dtype=torch.int32, device="cuda")
    out = []
    for shift in (0, 1):
        a = [_place(t, shift) for t in (q, k, v, cos, sin)]
        kc, vc = (_place(torch.zeros(2, kvh, cap, hd, dtype=torch.bfloat16, device="cuda"), shift) for _ in range(2))
        _lib.check(lib.lbk_rope_kv_append_rows(ctx.handle, *[t.data_ptr() for t in a], pos.data_ptr(), n, nh, kvh, hd, cap, seq, kc.data_ptr(), vc.data_ptr(), st))
        out.append((a[0], kc, vc))
    assert all(torch.equal(x, y) for x, y in zip(*out))
    ctx.check_device_error()
    c, s, half = cos[pos0:pos0 + n, None].double(), sin[pos0:pos0 + n, None].double(), hd // 2

    def turn(x):
        x = x.double()
        other = torch.cat([-x[..., half:], x[..., :half]], -1)
        return x * c + other * s, (x * c).abs() + (other * s).abs()

    got, kc, vc = out[0]
    want, size = turn(q)
    assert bool(((got.double() - want).abs() <= 2.0 ** -23 * size).all())  # a product and the sum, each rounded once: 2^-24 of each
    want, size = turn(k)
    new = slice(pos0, pos0 + n)
    assert bool(((kc[seq, :, new].transpose(0, 1).double() - want).abs() <= 2.0 ** -23 * size + 2.0 ** -8 * want.abs()).all())
    assert torch.equal(vc[seq, :, new].transpose(0, 1), v.to(torch.bfloat16))
    assert not kc[0].any() and not kc[1, :, :pos0].any() and not kc[1, :, pos0 + n:].any()
