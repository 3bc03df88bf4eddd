"""A prompt of which few places are wanted: the last layer works on those rows alone, and neither their logits nor what the prompt leaves in the cache
depend on it. Prompts around the sizes at which another form takes over (tiles of 128 rows, 64 rows, 32, 9 and 8), portions, every family."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VOCAB = 96


@pytest.fixture(scope="module")
def models(ctx, tmp_path_factory):
    from lemonade_burn_b200 import dugulorn, model, pefolix
    out = {}
    d = tmp_path_factory.mktemp("bitnet")
    cfg = model.Config(512, 768, 4, 1, 2, VOCAB, 1e-5, 500000.0, 2048)
    model.save_checkpoint(d, cfg, model.random_checkpoint(cfg, 3))
    out["bitnet"] = model.NativeBitNet(d, ctx)
    a = pefolix.attention_layer
    for name, mlp in (("pefolix", pefolix.dense_mlp(640)), ("experts", pefolix.moe_mlp(16, 3, 128, 192))):
        d = tmp_path_factory.mktemp(name)
        c = pefolix.make_config(VOCAB, 512, [a(4, 1, 128, 128, 64 if i else None, 2 if i else 0, None, mlp) for i in range(2)])
        pefolix.save_checkpoint(d, c, pefolix.random_checkpoint(c, 5))
        out[name] = pefolix.NativePefolix(d, ctx)
    kinds = {"lightning": dugulorn.lightning_layer(4, 128, 128, [0.9, 0.95, 0.99, 0.5], 640), "delta": dugulorn.delta_layer(4, 4, 128, 128, 4, 640),
             "latent": dugulorn.latent_layer(4, 128, 64, 128, 192, 128, None, 1e4, None, None, 640)}
    shared = dugulorn.latent_layer(4, 128, 64, 128, 192, 128, None, 1e4, None, 0, 640)
    for name, layers in {"lightning": [kinds["latent"], kinds["lightning"]], "delta": [kinds["latent"], kinds["delta"]], "latent": [kinds["delta"], kinds["latent"]],
                         "shared": [kinds["latent"], shared]}.items():
        d = tmp_path_factory.mktemp(name)
        c = dugulorn.make_config(VOCAB, 512, layers)
        dugulorn.save_checkpoint(d, c, dugulorn.random_checkpoint(c, 7))
        out[name] = dugulorn.NativeDugulorn(d, ctx)
    return out


@pytest.mark.parametrize("family", ["bitnet", "pefolix", "experts", "lightning", "delta", "latent", "shared"])
@pytest.mark.parametrize("n,want", [(5, [4]), (12, [2, 11]), (40, [39]), (63, [62]), (130, [129]), (130, [127, 128]), (300, [299]), (300, [140, 299, 200]), (300, [])])
def test_wanted_rows(models, ctx, family, n, want):
    import torch
    net = models[family]
    rng = np.random.default_rng(n)
    tokens = rng.integers(0, VOCAB, n + 3).astype(np.uint32)
    caches = [net.new_cache(2, 400) for _ in range(2)]
    # sequence 1, once with all rows and once with the wanted ones only; then a second portion and decode steps on both
    full = net.forward_rows(tokens[:n], caches[0], list(range(n)), seq=1)
    few = net.forward_rows(tokens[:n], caches[1], want, seq=1)
    spread = float(np.abs(full).max())
    # bf16 sums in another order; a turned code of the ternary model's quantisers moves a row by a few per mille of its spread (0.009 at most, measured on such models)
    tol = (2e-2 if family != "bitnet" else 1e-2) * spread
    if want:
        assert np.abs(few - full[want]).max() <= tol
    after = [net.forward_rows(tokens[n:n + 2], c, [0, 1], seq=1) for c in caches]
    assert np.abs(after[0] - after[1]).max() <= 1e-6 * spread, "the cache depends on the places that were wanted"
    step = torch.tensor([1, int(tokens[n + 2])], dtype=torch.int32, device="cuda")
    logits = [net.decode(step, c)[0] for c in caches]
    assert float((logits[0] - logits[1]).abs().max()) <= 1e-6 * spread
    ctx.check_device_error()


@pytest.mark.parametrize("inner", [6912, 8196])
def test_memory_of_a_prompt(ctx, tmp_path, inner):
    """What a prompt's first pass allocates: one row of the feed-forward width for each token where gate and up leave the GEMM as one, three where the width
    is beyond what the norm quantises (8192), and the rest; and short prompts, which go by other kernels, behind long ones and in front of them."""
    import torch
    from lemonade_burn_b200 import model
    n, hidden = 4096, 512
    cfg = model.Config(hidden, inner, 4, 1, 2, VOCAB, 1e-5, 500000.0, 4200)
    model.save_checkpoint(tmp_path, cfg, model.random_checkpoint(cfg, 3))
    net = model.NativeBitNet(tmp_path, ctx)
    cache = net.new_cache(2, 4200)
    tokens = np.random.default_rng(1).integers(0, VOCAB, n + 30).astype(np.uint32)
    early = net.forward_rows(tokens[:7], cache, [6], seq=1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    net.forward_rows(tokens[:n], cache, [n - 1])
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    rows = 3 if inner > 8192 else 1
    assert taken <= n * (rows * inner * 4 + 7 * hidden * 4 + inner) + (64 << 20), taken
    for k in (8, 9, 10):  # the last layer's rows alone, on both sides of the line
        net.reset_cache(cache)
        few = net.forward_rows(tokens[:30], cache, list(range(30 - k, 30)))
        net.reset_cache(cache)
        full = net.forward_rows(tokens[:30], cache, list(range(30)))
        assert np.abs(few - full[30 - k:]).max() <= 1e-2 * np.abs(full).max()
    net.reset_cache(cache)
    assert np.array_equal(net.forward_rows(tokens[:7], cache, [6], seq=1), early)
    ctx.check_device_error()
