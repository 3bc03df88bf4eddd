"""The quantiser around the row lengths at which another form takes over (3, 4 and 7 float4 a thread of 256, 8 of 512, rows read twice), aligned and
not, against the oracle: codes, scales and sums are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [4, 3068, 3072, 3076, 4096, 4100, 7168, 7172, 16384, 16388, 130, 2559])
@pytest.mark.parametrize("shift", [0, 1])
def test_row_lengths(oracle, ctx, k, shift):
    import torch
    from lemonade_burn_b200 import _lib
    m = 3
    rng = np.random.default_rng(k)
    x = (rng.standard_normal((m, k)) * np.array([[1.0], [1e-7], [50.0]])).astype(np.float32)
    x[0, k // 2] = np.nan
    buf = torch.zeros(m * k + 4, dtype=torch.float32, device="cuda")
    xd = buf[shift:shift + m * k]
    xd.copy_(torch.from_numpy(x.reshape(-1)))
    kp = -(-k // 128) * 128
    q = torch.full((m, kp), 77, dtype=torch.int8, device="cuda")
    s, t = torch.zeros(m, device="cuda"), torch.zeros(m, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().lbk_quantize_acts_dev(ctx.handle, xd.data_ptr(), m, k, q.data_ptr(), s.data_ptr(), t.data_ptr(), torch.cuda.current_stream().cuda_stream))
    wq, ws, wt = oracle.quantize_acts(x)
    assert np.array_equal(q.cpu().numpy()[:, :k], np.asarray(wq).reshape(m, -1)[:, :k])
    assert not q[:, k:].any()
    assert np.array_equal(s.cpu().numpy().view(np.uint32), np.asarray(ws, dtype=np.float32).view(np.uint32))
    assert np.array_equal(t.cpu().numpy(), np.asarray(wt))
    ctx.check_device_error()


@pytest.mark.parametrize("m", [1, 700])
@pytest.mark.parametrize("k", [7172, 8192, 8196, 12288, 12292, 20000, 21004, 28673])
def test_long_rows(oracle, ctx, m, k):
    """Where one form ends and the next begins, and rows that are read twice, whole units and not, few and more than the SMs hold."""
    import torch
    from lemonade_burn_b200 import _lib
    rng = np.random.default_rng(k + m)
    x = (rng.standard_normal((m, k)) * np.exp(rng.standard_normal((m, 1)))).astype(np.float32)
    if m > 1:
        x[3] = 0
        x[5, k - 1] = 1e6  # the maximum in the last column
    xd, kp = torch.from_numpy(x).cuda(), -(-k // 128) * 128
    q = torch.full((m, kp), 77, dtype=torch.int8, device="cuda")
    s, t = torch.empty(m, device="cuda"), torch.empty(m, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().lbk_quantize_acts_dev(ctx.handle, xd.data_ptr(), m, k, q.data_ptr(), s.data_ptr(), t.data_ptr(), torch.cuda.current_stream().cuda_stream))
    rows = slice(None) if m == 1 else slice(0, 9)
    qw, sw, tw = oracle.quantize_acts(x[rows])
    assert np.array_equal(q[rows, :k].cpu().numpy(), np.asarray(qw)[:, :k]) and np.array_equal(t[rows].cpu().numpy(), tw)
    assert np.array_equal(s[rows].cpu().numpy().view(np.uint32), np.asarray(sw, dtype=np.float32).view(np.uint32))
    assert not bool(q[:, k:].any()) and torch.equal(q.int().sum(1, dtype=torch.int32), t)
    ctx.check_device_error()
