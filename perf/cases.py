"""The framework's work, as cases that can be timed and checked: what a program that uses it has it do.

A case is a dict of plain values. `prepare` makes what such a program holds before the call (weights from the seed, a plan or
a loaded model with its cache, inputs), `run` is one pass through the public entry points, `exact` is the same result from
plain torch in 64 bits, `work` is the least a pass has to read, write and compute.

Kinds:

    linear    one group of packed ternary projections on m token rows (`ops.ternary_linear_multi`): the operator boundary that
              a decoder written elsewhere calls. 1 to 16 rows is decoding, more is a batch of prompts.
    sweep     a recorded plan of all projections of a model, one token (`ops.Plan`): the weight stream of a decode step.
    bitnet, pefolix, dugulorn
              a loaded model: prompts of `batch` sequences into one cache, then `steps` recorded decode steps that replay given
              tokens (scoring a continuation: the same work as generating it, with a result that does not hang on ties).
              `steps` 0 is a prompt pass by itself, with the logits of its last places.

Sizes: 2560 wide with 20 heads and 6912 in the feed-forward is the 2B4T shape, 4096 with 32 and 14336 the wider one that the
benchmarks of all families use; prompts and batches are those of a chat or of a small server.
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch

HEAD = 128              # size of an attention head
LAST = 8                # places of a prompt pass whose logits are asked for
WIDTHS = {2560: 6912, 4096: 14336}   # width -> feed-forward
Q_RANK, KV_RANK, ROT, TAPS, LOW = 1536, 512, 64, 4, 128
EXPERTS, TOP, EXPERT_FF, SHARED_FF = 64, 6, 1408, 2816
KEEP_FIRST = 4
EPS = {"bitnet": 1e-5, "pefolix": 1e-6, "dugulorn": 1e-6}


# ---- the cases ----------------------------------------------------------------------------------

def linear(part: str, width: int, m: int, ff: int = 0, name: str = "") -> dict:
    return {"name": name, "kind": "linear", "part": part, "width": width, "ff": ff or WIDTHS[width], "m": m}


def sweep(width: int, layers: int, name: str = "") -> dict:
    return {"name": name, "kind": "sweep", "width": width, "ff": WIDTHS[width], "layers": layers}


def model(kind: str, width: int, layers: int, vocab: int, batch: int, prompt: int, steps: int, window: int = 0, experts: bool = False, name: str = "") -> dict:
    return {"name": name, "kind": kind, "width": width, "ff": WIDTHS[width], "layers": layers, "vocab": vocab, "batch": batch, "prompt": prompt,
            "steps": steps, "window": window, "experts": experts}


def listed() -> list:
    return [
        # one token through q/k/v: the smallest call, all latency
        linear("qkv", 2560, 1, name="linear qkv 1 row"),
        # a decode batch of eleven through gate and up
        linear("gate_up", 2560, 11, name="linear gate/up 11 rows"),
        # a short prompt, its length a multiple of nothing, through the long projection
        linear("down", 2560, 333, name="linear down 333 rows"),
        # a long prompt through the largest group
        linear("gate_up", 2560, 2048, name="linear gate/up 2048 rows"),
        # every projection of a 2B4T-shaped model, one token
        sweep(2560, 30, name="sweep of 30 layers"),
        # a chat of one user: the whole 2B4T-shaped model, 2000 tokens read, 48 written
        model("bitnet", 2560, 30, 128256, 1, 2000, 48, name="bitnet chat"),
        # a server's batch: sixteen users with prompts of unequal length, 32 tokens each
        model("bitnet", 2560, 8, 32000, 16, 400, 32, name="bitnet batch of 16"),
        # reading a document of an odd length
        model("bitnet", 2560, 8, 32000, 1, 2011, 0, name="bitnet prompt"),
        # a long conversation under a sliding window
        model("pefolix", 2560, 4, 32000, 1, 3000, 48, window=1024, name="pefolix chat window"),
        # eight users of a model with experts
        model("pefolix", 2560, 2, 32000, 8, 200, 32, experts=True, name="pefolix batch of 8 experts"),
        # reading a document with recurrent and latent layers
        model("dugulorn", 2560, 4, 32000, 1, 2048, 0, name="dugulorn prompt"),
        # sixteen users of such a model
        model("dugulorn", 2560, 4, 32000, 16, 150, 48, name="dugulorn batch of 16"),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng) -> dict:
    kind = rng.choice(["linear", "linear", "linear", "sweep", "bitnet", "bitnet", "pefolix", "dugulorn", "dugulorn"])
    width = rng.choice([2560, 4096])
    if kind == "linear":
        ff = WIDTHS[width]
        if rng.random() < 0.5:  # sizes that are multiples of nothing
            width = _log(rng, 512, 4096)
            ff = round(width * rng.uniform(2.0, 3.5))
        case = linear(rng.choice(["qkv", "o", "gate_up", "down"]), width, _log(rng, 1, 2048), ff)
    elif kind == "sweep":
        case = sweep(width, _log(rng, 1, 30 if width == 2560 else 8))
    else:
        experts = kind == "pefolix" and rng.random() < 0.4
        if kind == "bitnet":
            layers = rng.randint(2, 8) if width == 2560 else rng.randint(1, 4)
        else:
            layers = (4 if kind == "dugulorn" else rng.randint(1, 4)) if width == 2560 else 1
        if experts:
            width, layers = 2560, rng.randint(1, 2)
        batch, prompt = _log(rng, 1, 16), _log(rng, 1, 2048)
        steps = 0 if rng.random() < 0.35 else _log(rng, 8, 48)
        if steps == 0:
            batch, prompt = 1, max(prompt, 16)
        prompt = min(prompt, 4096 // batch)
        case = model(kind, width, layers, 32000, batch, prompt, steps, rng.choice([0, 512, 1024]) if kind == "pefolix" else 0, experts)
    del case["name"]
    return case


# ---- sizes --------------------------------------------------------------------------------------

def _group(part: str, width: int, ff: int):
    """(columns, rows of each matrix) of a projection group; four query heads share a key head."""
    kv = width // 4
    return {"qkv": (width, [width, kv, kv]), "o": (width, [width]), "gate_up": (width, [ff, ff]), "down": (ff, [width])}[part]


PARTS = ("qkv", "o", "gate_up", "down")


def _lengths(case) -> list:
    """Prompt lengths of the sequences: unequal, the longest first."""
    return [max(1, case["prompt"] - 7 * s) for s in range(case["batch"])]


def _capacity(case) -> int:
    return case["prompt"] + case["steps"] + 1


def _dugulorn_kinds(case) -> list:
    return [("lightning", "latent", "delta", "shared")[i % 4] for i in range(case["layers"])]


def _decays(heads: int) -> list:
    return [0.5 + 0.499 * h / heads for h in range(heads)]


def _pefolix_experts(case, layer: int) -> bool:
    return bool(case["experts"]) and layer == case["layers"] - 1


def _shapes(case):
    """(tensor name, shape) of a bf16 family's checkpoint, in file order."""
    W, F, V, H = case["width"], case["ff"], case["vocab"], case["width"] // HEAD
    G, inner = H // 4, H * HEAD
    yield "embed", (V, W)
    if case["kind"] == "pefolix":
        for i in range(case["layers"]):
            p = f"l{i}."
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                yield p + n, (W,)
            yield p + "mix.q", (inner, W)
            yield p + "mix.k", (G * HEAD, W)
            yield p + "mix.v", (G * HEAD, W)
            yield p + "mix.o", (W, inner)
            if not _pefolix_experts(case, i):
                yield p + "mlp.gate", (F, W)
                yield p + "mlp.up", (F, W)
                yield p + "mlp.down", (W, F)
                continue
            for e in range(EXPERTS):
                yield f"{p}mlp.e{e}.up", (EXPERT_FF, W)
                yield f"{p}mlp.e{e}.down", (W, EXPERT_FF)
            yield p + "mlp.router", (EXPERTS, W)
            yield p + "mlp.shared.up", (SHARED_FF, W)
            yield p + "mlp.shared.down", (W, SHARED_FF)
            yield p + "mlp.shared.sg", (1, W)
        yield "final.norm", (W,)
        yield "head", (V, W)
        return
    yield "embed.norm", (W,)
    for i, kind in enumerate(_dugulorn_kinds(case)):
        p = f"l{i}."
        yield p + "norm1", (W,)
        yield p + "norm2", (W,)
        if kind in ("latent", "shared"):
            yield p + "mix.dq", (Q_RANK, W)
            yield p + "mix.dq.norm", (Q_RANK,)
            yield p + "mix.uq", (H * (HEAD + ROT), Q_RANK)
            if kind == "latent":
                yield p + "mix.dkv", (KV_RANK + ROT, W)
                yield p + "mix.dkv.norm", (KV_RANK,)
            yield p + "mix.uk", (inner, KV_RANK)
            yield p + "mix.uv", (inner, KV_RANK)
            yield p + "mix.g", (H, W)
        elif kind == "lightning":
            for n in ("q", "k", "v", "g"):
                yield p + "mix." + n, (inner, W)
            yield p + "mix.norm", (inner,)
        else:
            for n in ("q", "k", "v"):
                yield p + "mix." + n, (inner, W)
                yield p + f"mix.{n}.conv", (inner, TAPS)
            yield p + "mix.b", (H, W)
            yield p + "mix.A_log", (H,)
            yield p + "mix.norm", (HEAD,)
            yield p + "mix.a1", (LOW, W)
            yield p + "mix.a2", (inner, LOW)
            yield p + "mix.dt_bias", (inner,)
            yield p + "mix.g1", (LOW, W)
            yield p + "mix.g2", (inner, LOW)
        yield p + "mix.o", (W, inner)
        yield p + "mlp.up", (F, W)
        yield p + "mlp.up.b", (F,)
        yield p + "mlp.down", (W, F)
        yield p + "mlp.down.b", (W,)
    yield "final.norm", (W,)


# ---- weights and inputs from the seed -------------------------------------------------------------

def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _packed(gen, rows: int, cols: int):
    """Packed rows of i.i.d. ternary weights, zero with probability 0.4 (codes: two bits, weight + 1; rows end in zeros up to a
    multiple of 128)."""
    r = torch.rand((rows, -(-cols // 128) * 128), generator=gen, device="cuda")
    code = (r >= 0.3).to(torch.uint8) + (r >= 0.7).to(torch.uint8)
    code[:, cols:] = 1
    code = code.reshape(rows, -1, 4, 32)
    return (code[:, :, 0] | code[:, :, 1] << 2 | code[:, :, 2] << 4 | code[:, :, 3] << 6).reshape(rows, -1)


def _unpacked(packed, cols: int):
    """The weights of packed rows, in 64 bits."""
    b = packed.reshape(packed.shape[0], -1, 1, 32)
    shift = torch.tensor([0, 2, 4, 6], dtype=torch.uint8, device="cuda").reshape(1, 1, 4, 1)
    return ((b >> shift) & 3).reshape(packed.shape[0], -1)[:, :cols].double() - 1.0


def _scales(seed: int, n: int) -> list:
    """One per matrix, near 1 / mean |N(0, 0.02)| (32-bit values)."""
    return [float(v) for v in (60.0 + 5.0 * np.random.default_rng(seed).random(n)).astype(np.float32)]


def _linear_weights(case, seed):
    cols, rows = _group(case["part"], case["width"], case["ff"])
    gen = _generator(seed)
    packed = [_packed(gen, r, cols) for r in rows]
    x = torch.randn((case["m"], cols), generator=gen, device="cuda")
    return cols, packed, _scales(seed, len(rows)), x


def _sweep_weights(case, seed):
    """[(columns, packed matrices, scales, input row)] of every group of every layer."""
    gen, out = _generator(seed), []
    scales = iter(_scales(seed, 7 * case["layers"]))
    for _ in range(case["layers"]):
        for part in PARTS:
            cols, rows = _group(part, case["width"], case["ff"])
            out.append((cols, [_packed(gen, r, cols) for r in rows], [next(scales) for _ in rows], torch.randn((1, cols), generator=gen, device="cuda")))
    return out


BITNET_LINEARS = (("self_attn.q_proj", "qkv", 0), ("self_attn.k_proj", "qkv", 1), ("self_attn.v_proj", "qkv", 2), ("self_attn.o_proj", "o", 0),
                  ("mlp.gate_proj", "gate_up", 0), ("mlp.up_proj", "gate_up", 1), ("mlp.down_proj", "down", 0))


def _bitnet_weights(case, seed):
    """A stream that the embedding carries and to which every sublayer adds a little, as in a trained model: the gains of the
    norms in front of the last projections of the sublayers are small."""
    gen, W, F = _generator(seed), case["width"], case["ff"]
    scales = iter(_scales(seed, 7 * case["layers"]))
    t = {}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, part, k in BITNET_LINEARS:
            cols, rows = _group(part, W, F)
            t[p + name + ".qweight"] = _packed(gen, rows[k], cols)
            t[p + name + ".wscale"] = torch.tensor([next(scales)], dtype=torch.float32)
        for name, n, gain in (("input_layernorm", W, 1.0), ("post_attention_layernorm", W, 1.0), ("self_attn.attn_sub_norm", W, 0.05), ("mlp.ffn_sub_norm", F, 0.05)):
            t[p + name + ".weight"] = gain * (1.0 + 0.05 * torch.randn(n, generator=gen, device="cuda"))
    t["model.norm.weight"] = 1.0 + 0.05 * torch.randn(W, generator=gen, device="cuda")
    t["model.embed_tokens.weight"] = torch.randn((case["vocab"], W), generator=gen, device="cuda").to(torch.bfloat16)
    return t


def _bf16_weights(case, seed):
    """Matrices N(0, 1 / columns), embedding N(0, 1), norm weights near their neutral value, decays between none and strong."""
    gen, t = _generator(seed), {}
    near_zero = case["kind"] == "dugulorn"  # that family stores layer and model norms around zero
    for name, shape in _shapes(case):
        a = torch.randn(shape, generator=gen, device="cuda")
        if near_zero and (name.endswith((".norm1", ".norm2")) or name in ("embed.norm", "final.norm")):
            a *= 0.1
        elif name.endswith("A_log"):
            a *= 0.7
        elif name.endswith("dt_bias"):
            a = 1.5 * a - 2.0
        elif name.endswith(".b") and len(shape) == 1:
            a *= 0.3
        elif len(shape) == 1:
            a = 1.0 + 0.1 * a
        elif name != "embed":
            a *= shape[1] ** -0.5
        t[name] = a.to(torch.bfloat16)
    return t


def _tokens(case, seed) -> list:
    """Token ids of every sequence: its prompt and the continuation that is replayed."""
    rng = np.random.default_rng(seed + 1)
    return [rng.integers(0, case["vocab"], size=n + case["steps"]).astype(np.uint32) for n in _lengths(case)]


# ---- what a program has in hand, and one pass -------------------------------------------------------

def _load(case, seed):
    """The model, through a checkpoint folder as a program finds it."""
    from lemonade_burn_b200 import dugulorn, model as bitnet, pefolix
    W, F, L, V, H, kind = case["width"], case["ff"], case["layers"], case["vocab"], case["width"] // HEAD, case["kind"]
    with tempfile.TemporaryDirectory() as d:
        if kind == "bitnet":
            cfg = bitnet.Config(W, F, H, H // 4, L, V, EPS[kind], 500000.0, 4352)
            bitnet.save_checkpoint(d, cfg, {k: v.cpu() for k, v in _bitnet_weights(case, seed).items()})
            return bitnet.NativeBitNet(d)
        bits = {k: v.cpu().view(torch.int16).numpy().view(np.uint16) for k, v in _bf16_weights(case, seed).items()}
        if kind == "pefolix":
            layers = [pefolix.attention_layer(H, H // 4, HEAD, HEAD, case["window"] or None, KEEP_FIRST if case["window"] else 0, None,
                                              pefolix.moe_mlp(EXPERTS, TOP, EXPERT_FF, SHARED_FF) if _pefolix_experts(case, i) else pefolix.dense_mlp(F))
                      for i in range(L)]
            pefolix.save_checkpoint(d, pefolix.make_config(V, W, layers, EPS[kind]), bits)
            return pefolix.NativePefolix(d)
        layers = []
        for i, what in enumerate(_dugulorn_kinds(case)):
            if what == "lightning":
                layers.append(dugulorn.lightning_layer(H, HEAD, HEAD, _decays(H), F))
            elif what == "delta":
                layers.append(dugulorn.delta_layer(H, H, HEAD, HEAD, TAPS, F))
            else:
                layers.append(dugulorn.latent_layer(H, HEAD, ROT, HEAD, Q_RANK, KV_RANK, None, 1e6, dugulorn.yarn(4.0, 4096), i - 2 if what == "shared" else None, F))
        dugulorn.save_checkpoint(d, dugulorn.make_config(V, W, layers, EPS[kind]), bits)
        return dugulorn.NativeDugulorn(d)


def prepare(case: dict, seed: int) -> dict:
    from lemonade_burn_b200 import ops
    if case["kind"] == "linear":
        cols, packed, scales, x = _linear_weights(case, seed)
        return {"kind": "linear", "x": x, "linears": [ops.TernaryLinear(p, s, cols) for p, s in zip(packed, scales)]}
    if case["kind"] == "sweep":
        groups = _sweep_weights(case, seed)
        out = torch.empty(sum(p.shape[0] for _, packed, _, _ in groups for p in packed), dtype=torch.float32, device="cuda")
        plan, at = ops.Plan(), 0
        for cols, packed, scales, x in groups:
            linears = [ops.TernaryLinear(p, s, cols) for p, s in zip(packed, scales)]
            views = []
            for l in linears:
                views.append(out[at:at + l.rows])
                at += l.rows
            plan.add(x, linears, views)
        plan.finalize()
        return {"kind": "sweep", "plan": plan, "out": out}
    net = _load(case, seed)
    tokens = _tokens(case, seed)
    prompts = [t[:len(t) - case["steps"]] for t in tokens]
    replay = torch.from_numpy(np.stack([t[len(t) - case["steps"]:] for t in tokens], 1).astype(np.int32)).cuda()  # [steps, batch]
    want = [[len(p) - 1] if case["steps"] else list(range(max(0, len(p) - LAST), len(p))) for p in prompts]
    return {"kind": "model", "net": net, "cache": net.new_cache(case["batch"], _capacity(case)), "prompts": prompts, "want": want, "replay": list(replay)}


def run(state: dict):
    if state["kind"] == "linear":
        from lemonade_burn_b200 import ops
        return ops.ternary_linear_multi(state["x"], state["linears"])
    if state["kind"] == "sweep":
        state["plan"].run()
        return state["out"]
    net, cache = state["net"], state["cache"]
    net.reset_cache(cache)
    prompt = [net.forward_rows(p, cache, w, seq=s) for s, (p, w) in enumerate(zip(state["prompts"], state["want"]))]
    logits = [net.decode(t, cache)[0] for t in state["replay"]]
    return {"prompt": np.concatenate(prompt), "steps": torch.stack(logits) if logits else None}


# ---- the least a pass has to do ---------------------------------------------------------------------

def work(case: dict) -> dict:
    kind, W, F = case["kind"], case["width"], case["ff"]
    if kind == "linear":
        cols, rows = _group(case["part"], W, F)
        return {"bytes": sum(rows) * cols / 4 + case["m"] * (cols + sum(rows)) * 4, "flops": 2.0 * case["m"] * cols * sum(rows)}
    if kind == "sweep":
        groups = [_group(p, W, F) for p in PARTS] * case["layers"]
        return {"bytes": float(sum(sum(r) * c / 4 + (c + sum(r)) * 4 for c, r in groups)), "flops": float(sum(2 * c * sum(r) for c, r in groups))}
    H, G, L, V, steps, lens = W // HEAD, W // HEAD // 4, case["layers"], case["vocab"], case["steps"], _lengths(case)
    rows = sum(lens) + steps * case["batch"]                               # token rows through the layers
    heads = (case["batch"] + steps * case["batch"]) if steps else min(LAST, lens[0])   # rows through the head
    passes = len(lens) + steps                                             # times the weights are read
    cached = 0                                                             # positions of a layer's cache that decode steps read
    pairs = 0                                                              # query-key pairs of a layer
    for n in lens:
        for i in range(n + steps):
            seen = min(i + 1, case["window"] + KEEP_FIRST) if case["window"] else i + 1
            pairs += seen
            cached += seen if i >= n else 0
    if kind == "bitnet":
        params = sum(c * sum(r) for c, r in (_group(p, W, F) for p in PARTS))
        nbytes = passes * (L * params / 4 + V * W * 2) + L * cached * G * HEAD * 4
        flops = 2.0 * rows * L * params + 4.0 * L * pairs * H * HEAD
    elif kind == "pefolix":
        nbytes = flops = 0.0
        for i in range(L):
            attn, ff = W * HEAD * (2 * H + 2 * G), 3 * W * F
            read, used = ff, ff
            if _pefolix_experts(case, i):
                one, shared = 2 * W * EXPERT_FF, 2 * W * SHARED_FF
                used = TOP * one + shared
                read = sum(EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** n) for n in lens + [case["batch"]] * steps) * one / passes + shared
            nbytes += passes * (attn + read) * 2 + cached * G * HEAD * 4
            flops += 2.0 * rows * (attn + used) + 4.0 * pairs * H * HEAD
        nbytes += passes * V * W * 2
    else:
        nbytes, flops = passes * V * W * 2.0, 0.0
        matrices = {}
        for name, shape in _shapes(case):
            if len(shape) == 2 and name != "embed" and name.startswith("l"):
                matrices[name.split(".")[0]] = matrices.get(name.split(".")[0], 0) + shape[0] * shape[1]
        for i, what in enumerate(_dugulorn_kinds(case)):
            n = matrices[f"l{i}"]
            nbytes += passes * n * 2
            flops += 2.0 * rows * n
            if what in ("latent", "shared"):
                nbytes += cached * (KV_RANK + ROT) * 2
                flops += 2.0 * pairs * H * (2 * HEAD + ROT)
            else:
                nbytes += steps * case["batch"] * H * HEAD * HEAD * 8
                flops += rows * H * HEAD * HEAD * (7.0 if what == "delta" else 5.0)
    return {"bytes": float(nbytes + heads * V * 4), "flops": float(flops + 2.0 * heads * V * W)}


def tolerance(case: dict):
    """Against 64 bits the ternary decoder is 0.003 (8 layers) to 0.008 (30) off: codes of activations that lie on a rounding
    boundary turn with the last bit of any sum. The bf16 families are 0.003 to 0.006 off, 0.009 where a router's choice can turn."""
    if case["kind"] in ("linear", "sweep"):
        return "exact"      # whole numbers times one defined product of scales
    if case["kind"] == "bitnet" or case["experts"]:
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.02, "max": 0.2}


# ---- the same in 64 bits ------------------------------------------------------------------------------

def _quantized(x):
    """(whole codes, scale) of rows: 127 over the largest magnitude, ties to even."""
    scale = 127.0 / x.abs().amax(-1, keepdim=True).clamp_min(1e-5)
    return (x * scale).round().clamp(-128, 127), scale


def _ternary(x, packed, wscale):
    q, s = _quantized(x)
    return (q @ _unpacked(packed, x.shape[-1]).T) / (s * wscale)


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt((d * d).mean(-1, keepdim=True) + eps) * w


def _softmax_rows(q, k, v, scale, window=0, slopes=None):
    """q [n, H, d], k [n, G, d], v [n, G, e] -> [n, H * e], causal, head by head."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(n, device="cuda")
    dist = i[:, None] - i[None, :]
    see = dist >= 0
    if window:
        see &= (dist < window) | (i[None, :] < KEEP_FIRST)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if slopes is not None:
            s = s - slopes[h] * dist
        out.append(torch.softmax(s.masked_fill(~see, -math.inf), -1) @ v[:, h * G // H])
    return torch.cat(out, 1)


def _bitnet_exact(case, t, tokens):
    W, H, eps, n = case["width"], case["width"] // HEAD, EPS["bitnet"], len(tokens)
    inv = torch.from_numpy(np.array([1.0 / 500000.0 ** (2 * i / HEAD) for i in range(HEAD // 2)]).astype(np.float32))
    angle = (torch.arange(n, dtype=torch.float32)[:, None] * inv[None, :]).double().cuda()  # the model defines its angles in 32 bits
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]

    def turn(x):
        a, b = x[..., :HEAD // 2], x[..., HEAD // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    emb = t["model.embed_tokens.weight"]
    x = emb[torch.from_numpy(tokens.astype(np.int64)).cuda()].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        lin = lambda name, y: _ternary(y, t[p + name + ".qweight"], float(t[p + name + ".wscale"]))  # noqa: E731
        norm = lambda name, y: _rms(y, t[p + name + ".weight"].double(), eps)  # noqa: E731
        h = norm("input_layernorm", x)
        q, k, v = (lin(f"self_attn.{c}_proj", h).reshape(n, -1, HEAD) for c in "qkv")
        k, v = (y.to(torch.bfloat16).double() for y in (turn(k), v))  # the cache holds bf16
        x = x + lin("self_attn.o_proj", norm("self_attn.attn_sub_norm", _softmax_rows(turn(q), k, v, HEAD ** -0.5)))
        h = norm("post_attention_layernorm", x)
        a = lin("mlp.gate_proj", h).clamp_min(0) ** 2 * lin("mlp.up_proj", h)
        x = x + lin("mlp.down_proj", norm("mlp.ffn_sub_norm", a))
    return _rms(x, t["model.norm.weight"].double(), eps), emb


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _pefolix_exact(case, t, tokens):
    W, H, eps, n = case["width"], case["width"] // HEAD, EPS["pefolix"], len(tokens)
    w = lambda name: t[name].double()  # noqa: E731
    slopes = [2.0 ** (-8.0 * (h + 1) / H) for h in range(H)]
    x = t["embed"][torch.from_numpy(tokens.astype(np.int64)).cuda()].double()
    for i in range(case["layers"]):
        p = f"l{i}."
        h = _layer_norm(x, w(p + "norm1"), eps)
        q, k, v = ((h @ w(p + "mix." + c).T).reshape(n, -1, HEAD) for c in "qkv")
        y = _softmax_rows(q, k, v, HEAD ** -0.5, case["window"], slopes) @ w(p + "mix.o").T
        x = x + _layer_norm(y, w(p + "norm1b"), eps)
        h = _layer_norm(x, w(p + "norm2"), eps)
        if _pefolix_experts(case, i):
            score, ids = torch.softmax(h @ w(p + "mlp.router").T, -1).topk(TOP, -1)
            y = torch.sigmoid(h @ w(p + "mlp.shared.sg").T) * ((h @ w(p + "mlp.shared.up").T).clamp_min(0) ** 2 @ w(p + "mlp.shared.down").T)
            for e in range(EXPERTS):
                row, place = (ids == e).nonzero(as_tuple=True)
                if len(row):
                    y[row] += score[row, place, None] * ((h[row] @ w(f"{p}mlp.e{e}.up").T).clamp_min(0) ** 2 @ w(f"{p}mlp.e{e}.down").T)
        else:
            y = (_gelu(h @ w(p + "mlp.gate").T) * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
        x = x + _layer_norm(y, w(p + "norm2b"), eps)
    return _layer_norm(x, w("final.norm"), eps), t["head"]


def _rotated(x, factor=4.0, original=4096, base=1e6, fast=32.0, slow=1.0):
    """Neighbouring dimensions of x [n, heads, ROT] turned by position, with YaRN-scaled frequencies."""
    at = lambda turns: ROT * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(fast)), 0), min(math.ceil(at(slow)), ROT - 1)
    f = []
    for i in range(ROT // 2):
        ramp = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        one = base ** (-2.0 * i / ROT)
        f.append(one / factor * ramp + one * (1.0 - ramp))
    a = (torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None] * torch.tensor(f, device="cuda", dtype=torch.float64))[:, None, :]
    m = 0.1 * math.log(factor) + 1.0
    c, s = a.cos() * m, a.sin() * m
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).reshape(x.shape)


def _silu(z):
    return z * torch.sigmoid(z)


def _short_conv(x, taps):
    y = torch.zeros_like(x)
    for j in range(TAPS):
        back = TAPS - 1 - j
        y[back:] += x[:x.shape[0] - back] * taps[:, j]
    return y


def _recurrence(q, k, v, decay, beta=None):
    """q, k, v [n, H, 128], decay [n or 1, H, 128 or 1]: the state of every head token by token, with beta the delta rule's."""
    S = torch.zeros((q.shape[1], HEAD, HEAD), dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    for i in range(q.shape[0]):
        S = S * decay[i if decay.shape[0] > 1 else 0][:, :, None]
        u = v[i] if beta is None else beta[i][:, None] * (v[i] - torch.matmul(k[i][:, None, :], S)[:, 0])
        S.baddbmm_(k[i][:, :, None], u[:, None, :])
        out[i] = torch.matmul(q[i][:, None, :], S)[:, 0]
    return out


def _dugulorn_exact(case, t, tokens):
    H, eps, n = case["width"] // HEAD, EPS["dugulorn"], len(tokens)
    w = lambda name: t[name].double()  # noqa: E731
    x = _rms(t["embed"][torch.from_numpy(tokens.astype(np.int64)).cuda()].double(), 1.0 + w("embed.norm"), eps)
    latents = {}
    for i, kind in enumerate(_dugulorn_kinds(case)):
        p = f"l{i}.mix."
        lin = lambda name, y: y @ w(p + name).T  # noqa: E731
        heads = lambda y: y.reshape(n, H, -1)  # noqa: E731
        if kind in ("latent", "shared"):
            if kind == "latent":
                kv = lin("dkv", x)
                latents[i] = _rms(kv[:, :KV_RANK], w(p + "dkv.norm"), eps), _rotated(kv[:, None, KV_RANK:])
            c, kr = latents[i if kind == "latent" else i - 2]
            q = heads(lin("uq", _rms(lin("dq", x), w(p + "dq.norm"), eps)))
            q = torch.cat([q[..., :HEAD], _rotated(q[..., HEAD:])], -1)
            k = torch.cat([heads(lin("uk", c)), kr.expand(n, H, ROT)], -1)
            o = heads(_softmax_rows(q, k, heads(lin("uv", c)), (HEAD + ROT) ** -0.5)) * torch.sigmoid(lin("g", x))[:, :, None]
        elif kind == "lightning":
            q, k, v = (heads(_silu(lin(name, x))) for name in "qkv")
            o = _recurrence(q, k, v, torch.tensor(_decays(H), dtype=torch.float64, device="cuda").reshape(1, H, 1)).reshape(n, -1)
            o = _rms(o, w(p + "norm"), eps) * torch.sigmoid(lin("g", x))
        else:
            q, k, v = (heads(_silu(_short_conv(lin(name, x), w(f"{p}{name}.conv")))) for name in "qkv")
            q, k = (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
            step = torch.nn.functional.softplus(lin("a2", lin("a1", x)) + w(p + "dt_bias"), threshold=1e9)
            g = torch.exp(-torch.exp(w(p + "A_log"))[:, None] * heads(step))
            o = _rms(_recurrence(q * HEAD ** -0.5, k, v, g, torch.sigmoid(lin("b", x))), w(p + "norm"), eps)
            o = o * heads(torch.sigmoid(lin("g2", lin("g1", x))))
        x = x + _rms(lin("o", o.reshape(n, -1)), 1.0 + w(f"l{i}.norm1"), eps)
        m = f"l{i}.mlp."
        y = (x @ w(m + "up").T + w(m + "up.b")).clamp_min(0) ** 2 @ w(m + "down").T + w(m + "down.b")
        x = x + _rms(y, 1.0 + w(f"l{i}.norm2"), eps)
    return _rms(x, 1.0 + w("final.norm"), eps), t["embed"]


def exact(case: dict, seed: int):
    if case["kind"] == "linear":
        _, packed, scales, x = _linear_weights(case, seed)
        return [_ternary(x.double(), p, s) for p, s in zip(packed, scales)]
    if case["kind"] == "sweep":
        return torch.cat([_ternary(x.double(), p, s)[0] for _, packed, scales, x in _sweep_weights(case, seed) for p, s in zip(packed, scales)])
    weights = _bitnet_weights(case, seed) if case["kind"] == "bitnet" else _bf16_weights(case, seed)
    forward = {"bitnet": _bitnet_exact, "pefolix": _pefolix_exact, "dugulorn": _dugulorn_exact}[case["kind"]]
    steps, prompt, after = case["steps"], [], []
    for tokens in _tokens(case, seed):
        h, head = forward(case, weights, tokens)
        n = len(tokens) - steps
        logits = (h[n - 1:] if steps else h[max(0, n - LAST):]) @ head.double().T
        prompt.append(logits[:1] if steps else logits)
        after.append(logits[1:])
    return {"prompt": torch.cat(prompt), "steps": torch.stack(after, 1) if steps else None}
