"""Embedding rows around the width from which they go in units of four, widths that are no units, tables and outputs that do not lie on a unit. Equality."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [1, 96, 508, 511, 512, 514, 516, 2560, 2561, 8196])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("m", [3, 600])
def test_rows(ctx, m, hidden, shift):
    import torch
    from lemonade_burn_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(hidden + shift)
    table = torch.randn(37 * hidden + shift, generator=g, device="cuda").to(torch.bfloat16)[shift:].view(37, hidden)
    toks = torch.randint(0, 37, (m,), dtype=torch.int32, generator=g, device="cuda")
    for out_shift in (0, 1):
        out = torch.full((m * hidden + 1 + out_shift,), -7.0, device="cuda")
        got = out[out_shift:out_shift + m * hidden].view(m, hidden)
        _lib.check(_lib.load().lbk_embed_bf16(ctx.handle, table.data_ptr(), toks.data_ptr(), m, hidden, got.data_ptr(), torch.cuda.current_stream().cuda_stream))
        assert torch.equal(got, table[toks.long()].float())
        assert float(out[-1]) == -7.0 and (not out_shift or float(out[0]) == -7.0)
    ctx.check_device_error()
