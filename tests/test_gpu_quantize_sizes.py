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
