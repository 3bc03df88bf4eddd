"""Experts at up to sixteen tokens at the widths where the few-token kernels' boxes change: boxes of two tiles (18 rows an SM), several boxes of them,
more boxes than a warp carries at a time; more up tiles than a CTA carries at a time; warps that have none of the shared expert's columns
and warps that have none of the experts'. Against the Pefolix oracle in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SMS = 148
# width, experts, chosen, their feed-forward, the shared expert's (0: none)
MODELS = {
    "one box of two tiles, five up tiles a CTA": (2560, 24, 20, 500, 90),
    "the same without a shared expert": (2560, 24, 20, 500, 0),
    "two boxes, an odd width": (SMS * 32 + 5, 5, 2, 200, 130),
    "three boxes, twenty shared chunks and one of the expert": (SMS * 65, 3, 1, 60, 1270),
    "three boxes, a chunk an expert": (SMS * 65, 7, 3, 64, 0),
}
VOCAB = 256


@pytest.mark.parametrize("name", list(MODELS))
def test_few_token_experts(ctx, tmp_path, name):
    """Every word of the vocabulary looks at a run of neighbouring columns of its own, so that a box that went wrong shows in full. Tolerance: 2^-9 of
    a value for each of about eight roundings to bf16 on the way, which add up like their squares, is 0.0055 of the logits' spread; six times
    that over some thousand logits. A token whose choice of experts hangs on less than 0.05 of a router logit is left out."""
    from lemonade_burn_b200 import pefolix
    from oracle import pefolix_oracle as po
    width, experts, top, ff, shared = MODELS[name]
    cfg = pefolix.make_config(VOCAB, width, [pefolix.attention_layer(2, 1, 32, 32, None, 0, 0.2, pefolix.moe_mlp(experts, top, ff, shared or None))])
    t = pefolix.random_checkpoint(cfg, width + shared)
    rng = np.random.default_rng(1)
    head = np.zeros((VOCAB, width), np.float32)
    for v, cols in enumerate(np.array_split(np.arange(width), VOCAB)):
        head[v, cols] = rng.choice([-1.0, 1.0], size=len(cols)) * len(cols) ** -0.5
    t["head"] = pefolix.bf16_bits(head)
    pefolix.save_checkpoint(tmp_path, cfg, t)
    _, w = po.load(tmp_path)
    toks = rng.integers(0, VOCAB, size=34).astype(np.uint32)
    want = po.forward(cfg, w, toks)
    x = w["embed"][toks]
    h = po.layer_norm(x, w["l0.norm1"], cfg["norm"]["eps"])
    x = x + po.layer_norm(po.mixer(h, w, "l0.mix.", cfg["layers"][0]["mixer"], np.arange(len(toks))), w["l0.norm1b"], cfg["norm"]["eps"])
    z = -np.sort(-(po.layer_norm(x, w["l0.norm2"], cfg["norm"]["eps"]) @ w["l0.mlp.router"].T), axis=1)
    clear = np.ones(len(toks), bool) if top == experts else z[:, top - 1] - z[:, top] > 0.05
    assert clear.sum() >= 20
    net = pefolix.NativePefolix(tmp_path, ctx)
    c, at, got = net.new_cache(1, len(toks)), 0, []
    for n in (1, 8, 9, 16):
        got.append(net.forward(toks[at:at + n], c, all_logits=True))
        at += n
    err = np.abs(np.concatenate(got) - want) / want.std()
    assert err[clear].max() < 6 * 0.0055, (np.sort(err[clear].max(1))[-3:], np.argwhere(err == err[clear].max()))
    ctx.check_device_error()
    net.close()
