"""lbk_norm_quant at the row lengths where the number of values a thread holds changes: the bits of the norm kernel followed by the
quantiser."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 3068, 3072, 3076, 4096, 4100, 7168, 7172, 8188])
@pytest.mark.parametrize("pre", [1, 2, 3])
def test_norm_quant_at_the_edges(ctx, n, pre):
    import torch
    from lemonade_burn_b200 import _lib
    lib, st, rows, kp = _lib.load(), torch.cuda.current_stream().cuda_stream, 5, (n + 127) // 128 * 128
    g = torch.Generator(device="cuda").manual_seed(n)
    x, y = 3.0 * torch.randn(rows, n, generator=g, device="cuda"), torch.randn(rows, n, generator=g, device="cuda")
    w = torch.rand(n, generator=g, device="cuda") + 0.5
    x[1] = 0.0   # a row without values keeps the smallest scale
    xa, xb, f = x.clone(), x.clone(), torch.empty_like(x)
    args = (rows, n, 1e-5, f.data_ptr(), st)
    if pre == 1:
        _lib.check(lib.lbk_rms_norm(ctx.handle, xa.data_ptr(), w.data_ptr(), *args))
    else:
        op = lib.lbk_add_rms_norm if pre == 2 else lib.lbk_relu2_mul_rms_norm
        _lib.check(op(ctx.handle, xa.data_ptr(), y.data_ptr(), w.data_ptr(), *args))
    out = [(torch.full((rows, kp), 77, dtype=torch.int8, device="cuda"), torch.empty(rows, device="cuda"), torch.empty(rows, dtype=torch.int32, device="cuda"))
           for _ in range(2)]
    _lib.check(lib.lbk_quantize_acts_dev(ctx.handle, f.data_ptr(), rows, n, *[t.data_ptr() for t in out[0]], st))
    _lib.check(lib.lbk_norm_quant(ctx.handle, pre, xb.data_ptr(), y.data_ptr(), w.data_ptr(), rows, n, 1e-5, *[t.data_ptr() for t in out[1]], st))
    assert torch.equal(xa, xb) and all(torch.equal(a, b) for a, b in zip(*out))
    ctx.check_device_error()
