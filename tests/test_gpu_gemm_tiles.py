"""Prefill GEMM at the edges of its tiles: token rows around the narrow form's 64 and the wide form's 192, ragged last token tiles, K of one
block to several packed-weight stages (last stages of one, two and three blocks, whose second half or whole is one set of expanders' or nobody's),
row tiles of one to many, one to three matrices. Whole numbers: equality with the oracle. And launches close behind one another: the same rows every time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def group(oracle, ctx, rows, cols, m, seed):
    import torch
    from lemonade_burn_b200 import ops
    rng = np.random.default_rng(seed)
    packed = [oracle.pack_matrix(rng.choice(np.array([-1, 0, 1], dtype=np.int8), size=(r, cols), p=[0.3, 0.4, 0.3])) for r in rows]
    scales = [np.float32(50 + 3 * i) for i in range(len(rows))]
    x = rng.standard_normal((m, cols)).astype(np.float32)
    lins = [ops.TernaryLinear(torch.from_numpy(p).cuda(), float(s), cols, ctx) for p, s in zip(packed, scales)]
    return packed, scales, x, torch.from_numpy(x).cuda(), lins


@pytest.mark.parametrize("rows,cols", [([128], 128), ([300, 4], 640), ([256, 128, 77], 896), ([20000], 256)])
@pytest.mark.parametrize("m", [17, 63, 64, 65, 95, 97, 192, 193, 400, 577])
def test_tile_edges(oracle, ctx, rows, cols, m):
    from lemonade_burn_b200 import ops
    packed, scales, x, xd, lins = group(oracle, ctx, rows, cols, m, cols + m)
    q, s, ssum = oracle.quantize_acts(x)
    wf, wi = oracle.simd_gemm_multi(packed, scales, q, s, ssum, want_i32=True)
    outs, iouts = ops.ternary_linear_multi(xd, lins, want_i32=True)
    for got, goti, ef, ei in zip(outs, iouts, wf, wi):
        assert np.array_equal(goti.cpu().numpy(), ei)
        assert np.array_equal(got.cpu().numpy().view(np.uint32), ef.view(np.uint32))
    outs = ops.ternary_linear_multi(xd, lins)  # without integer outputs K may be cut into parts
    for got, ef in zip(outs, wf):
        assert np.array_equal(got.cpu().numpy().view(np.uint32), ef.view(np.uint32))
    ctx.check_device_error()


@pytest.mark.parametrize("m", [333, 2011])
def test_launches_behind_one_another_give_the_same_rows(oracle, ctx, m):
    """Weights that are overwritten in the ring before they are read turn up as single rows of a tile, once in thousands: 2011 rows
    of 2560 -> 2 x 6912, eight launches in a row with nothing between them, 40 times."""
    import torch
    from lemonade_burn_b200 import ops
    _, _, _, xd, lins = group(oracle, ctx, [6912, 6912], 2560, m, 7)
    want = [o.clone() for o in ops.ternary_linear_multi(xd, lins)]
    for _ in range(40):
        for outs in [ops.ternary_linear_multi(xd, lins) for _ in range(8)]:
            for a, b in zip(outs, want):
                assert torch.equal(a, b)
    ctx.check_device_error()


@pytest.mark.parametrize("cols,rows,m", [(8192, [2048, 2048], 777), (8640, [3200], 1024), (512, [1376, 1376], 2048), (1000, [2700, 2700], 256), (14336, [4096], 17), (14336, [4096], 61),
                                         (8192, [2048, 2048], 25), (20480, [1000], 150)])
def test_one_batch_or_portions(ctx, cols, rows, m):
    """Launches whose last round are short tiles, matrices of few columns, long columns in few tiles: whatever tile and cut are chosen for all rows at once, the
    bits are those of the rows in portions of 64 and fewer, which go by other tiles. Equality: the same integers and products of scales."""
    import torch
    from lemonade_burn_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(cols + m)
    lins = [ops.TernaryLinear(torch.randint(0, 3, (r, -(-cols // 128) * 32), generator=g, device="cuda", dtype=torch.uint8) * 21, 50.0 + i, cols, ctx) for i, r in enumerate(rows)]
    x = torch.randn(m, cols, generator=g, device="cuda")
    whole, ints = ops.ternary_linear_multi(x, lins, want_i32=True)
    for r0 in range(0, m, 64):
        part = ops.ternary_linear_multi(x[r0:r0 + 64], lins)
        for w, p in zip(whole, part):
            assert torch.equal(w[r0:r0 + 64], p)
    assert all(bool((i != 0).any()) for i in ints)
    ctx.check_device_error()
