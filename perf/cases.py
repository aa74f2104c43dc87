"""Performance cases: what programs have this framework do, through its public entry points.

Kinds of case:
  q4_layer       the four projections of one decoder layer on 4-bit weights (``quantize.gemm_tw_marlin``), `rows` rows at once
  q4_experts     one routed layer on 4-bit experts: ``batched_marlin_gate_up`` and ``batched_marlin_down_axpy``
  q4_generate    greedy decoding of the 4-bit decoder over a filled cache (``QuantizedGenerationEngine``)
  prompt         a whole prompt through a dense-weight decoder (``DenseEngine.step``), logits of its last token
  generate       a whole request of a dense-weight decoder (``DenseEngine.greedy``): prompt, then greedily decoded tokens

Sizes are those of ``bench.py``'s decoders.  Weights are random with trained-like structure where it matters for a comparison:
heads that predict clearly (so that greedy tokens do not hang on rounding) and routers that decide clearly (so that what
is nearly a tie at the cut carries little weight).
"""
from __future__ import annotations

import math
import zlib

import torch

from tensorwarp_b200 import dense, generate, quantize
from tensorwarp_b200.engine import DenseEngine
from tensorwarp_b200.models import bidasun, zukotar

DEV = "cuda"

# width, query heads, key/value heads, head size, feed-forward, vocabulary, window, kept first keys; experts, chosen, groups, kept
# groups, expert width, rotated part, latent, low rank; depth of the two dense-weight designs.  The depth of the two wide
# sizes is cut, so that weights are made in about a second.
SIZES = {
    "1b": dict(width=2048, heads=16, kv_heads=4, dim=128, ff=8192, vocab=32768, window=512, keep=4, experts=64, top=8, groups=8, kept=4,
               expert_ff=1024, rot=64, rank=512, low=16, depth={"bidasun": 16, "zukotar": 16, "q4": 16}),
    "7b": dict(width=3584, heads=28, kv_heads=4, dim=128, ff=18944, vocab=152064, window=1024, keep=4, experts=32, top=4, groups=4, kept=2,
               expert_ff=2560, rot=64, rank=512, low=16, depth={"bidasun": 14, "zukotar": 6, "q4": 28}),
    "13b-wide": dict(width=5120, heads=40, kv_heads=8, dim=128, ff=13824, vocab=32768, window=2048, keep=4, experts=16, top=2, groups=4, kept=2,
                     expert_ff=6144, rot=64, rank=512, low=32, depth={"bidasun": 6, "zukotar": 4, "q4": 12}),
}
TAU = 16.0
# as in a trained model, the stream is large beside what one layer adds: a choice of experts that rounding tips over stays a small matter
EMBED_SCALE = 8.0
THETA = 1e6


def listed():
    return [
        # one token through a layer as the reference's callers hold it: f32 rows, a scale for every 32 weights
        {"name": "q4_layer_1row_f32", "kind": "q4_layer", "size": "1b", "rows": 1, "dtype": "float32", "group": 32},
        # some twenty sequences decoding in lock step
        {"name": "q4_layer_24rows", "kind": "q4_layer", "size": "7b", "rows": 24, "dtype": "float16", "group": 128},
        # a prompt portion on 4-bit weights
        {"name": "q4_layer_200rows", "kind": "q4_layer", "size": "7b", "rows": 200, "dtype": "float16", "group": 128},
        # one token through a routed layer of 4-bit experts
        {"name": "q4_experts_top8", "kind": "q4_experts", "hidden": 2816, "ff": 704, "experts": 64, "top": 8, "group": 32},
        # one user's continuation on the 4-bit decoder, in the middle of a context
        {"name": "q4_7b_generate", "kind": "q4_generate", "size": "7b", "context": 2048, "new": 8},
        # a chat turn: a short prompt, where the weights are read once for a few rows
        {"name": "bidasun_1b_prompt_100", "kind": "prompt", "model": "bidasun", "size": "1b", "tokens": 100, "dtype": "bfloat16"},
        # a document: products of many rows, attention beyond the window
        {"name": "bidasun_7b_prompt_2048", "kind": "prompt", "model": "bidasun", "size": "7b", "tokens": 2048, "dtype": "bfloat16"},
        # a short answer to a short question
        {"name": "bidasun_1b_generate", "kind": "generate", "model": "bidasun", "size": "1b", "tokens": 37, "new": 24, "dtype": "bfloat16"},
        # the 32-bit option, as it is used to check a checkpoint
        {"name": "bidasun_1b_prompt_70_f32", "kind": "prompt", "model": "bidasun", "size": "1b", "tokens": 70, "dtype": "float32"},
        # a question with some context, on linear and latent layers with routed experts
        {"name": "zukotar_1b_prompt_333", "kind": "prompt", "model": "zukotar", "size": "1b", "tokens": 333, "dtype": "bfloat16"},
        # a document on the same model
        {"name": "zukotar_1b_prompt_4096", "kind": "prompt", "model": "zukotar", "size": "1b", "tokens": 4096, "dtype": "bfloat16"},
        # a short answer on the same model
        {"name": "zukotar_1b_generate", "kind": "generate", "model": "zukotar", "size": "1b", "tokens": 37, "new": 24, "dtype": "bfloat16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# longest drawn prompts: no more work than the largest listed case
LONGEST = {("bidasun", "1b"): 6000, ("bidasun", "7b"): 2000, ("bidasun", "13b-wide"): 3000, ("zukotar", "1b"): 6000, ("zukotar", "7b"): 4000,
           ("zukotar", "13b-wide"): 4000}


def draw(rng):
    kind = rng.choice(["q4_layer", "q4_layer", "q4_experts", "q4_generate", "prompt", "prompt", "prompt", "generate", "generate"])
    size = rng.choice(["1b", "7b", "13b-wide"])
    if kind == "q4_layer":
        f32 = rng.random() < 0.25
        return {"kind": kind, "size": size, "rows": _log(rng, 1, 8 if f32 else 256), "dtype": "float32" if f32 else "float16",
                "group": 32 if f32 else rng.choice([32, 128])}
    if kind == "q4_experts":
        return {"kind": kind, "hidden": 128 * rng.randint(4, 28), "ff": 64 * rng.randint(4, 40), "experts": rng.choice([16, 32, 64]),
                "top": rng.choice([2, 4, 6, 8]), "group": 32}
    if kind == "q4_generate":
        return {"kind": kind, "size": size, "context": _log(rng, 1, 3000), "new": rng.randint(3, 8)}
    model = rng.choice(["bidasun", "zukotar"])
    if model == "bidasun" and rng.random() < 0.15:
        return {"kind": "prompt", "model": model, "size": "1b", "tokens": _log(rng, 2, 256), "dtype": "float32"}
    if kind == "prompt":
        return {"kind": kind, "model": model, "size": size, "tokens": _log(rng, 2, LONGEST[model, size]), "dtype": "bfloat16"}
    case = {"kind": kind, "model": model, "size": size, "tokens": _log(rng, 1, 600), "new": rng.randint(4, 32), "dtype": "bfloat16"}
    while work(case)["bytes"] > 5e10:
        case["new"] -= 1
    return case


# ------------------------------------------------------------------------------------------------------ 4-bit layer --

def _generator(*key):
    return torch.Generator(device=DEV).manual_seed(zlib.crc32(repr(key).encode()))


def _layer_shapes(size):
    """(in, out) of the fused q|k|v, output, fused gate|up and down projections."""
    s = SIZES[size]
    q, kv = s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
    return [(s["width"], q + 2 * kv), (q, s["width"]), (s["width"], 2 * s["ff"]), (s["ff"], s["width"])]


def _packed(gen, k, n, group):
    """A quantised matrix as a checkpoint holds it: nibbles spread like rounded normal weights, f16 scales."""
    q = torch.randn((k // 32, n, 32), generator=gen, device=DEV).mul_(2.3).round_().add_(8).clamp_(0, 15).to(torch.uint8)
    packed = q[:, :, 0::2] | (q[:, :, 1::2] << 4)
    scales = (torch.rand((k // group, n), generator=gen, device=DEV) * 0.008 + 0.004).half()
    return packed.contiguous(), scales


def _unpacked(packed, scales, k, n, group):
    """The [k, n] weights in 64 bits."""
    p = packed.reshape(k // 32, n, 16)
    q = torch.stack((p & 15, p >> 4), dim=3).reshape(k // 32, n, 32).double().sub_(8)
    s = scales.reshape(k // group, n).double().repeat_interleave(group // 32, dim=0)
    return q.mul_(s[:, :, None]).permute(0, 2, 1).reshape(k, n)


def _prepare_q4_layer(case, seed):
    gen, dt = _generator("q4_layer", seed), getattr(torch, case["dtype"])
    m, g = case["rows"], case["group"]
    ops = []
    for k, n in _layer_shapes(case["size"]):
        packed, scales = _packed(gen, k, n, g)
        a = torch.randn((m, k), generator=gen, device=DEV).to(dt)
        ops.append((a, packed, scales, torch.zeros((m, n), dtype=dt, device=DEV), m, n, k))
    space = quantize.Workspace.for_shapes([(m, n, k, g) for k, n in _layer_shapes(case["size"])])
    return {"ops": ops, "group": g, "workspace": space}


def _run_q4_layer(state):
    for op in state["ops"]:
        quantize.gemm_tw_marlin(*op, group_size=state["group"], workspace=state["workspace"])
    return [op[3] for op in state["ops"]]


def _exact_q4_layer(case, state):
    return [a.double() @ _unpacked(packed, scales, k, n, state["group"]) for a, packed, scales, _, _, n, k in state["ops"]]


# ---------------------------------------------------------------------------------------------------- 4-bit experts --

def _prepare_q4_experts(case, seed):
    gen = _generator("q4_experts", seed)
    h, f, e, top, g = (case[x] for x in ("hidden", "ff", "experts", "top", "group"))
    up, down = _packed(gen, h, e * 2 * f, g), _packed(gen, f, e * h, g)

    def by_expert(t, n):                                                       # [.., experts * n, ..] -> expert after expert
        return t.reshape(t.shape[0], e, n, -1).transpose(0, 1).contiguous().reshape(-1)
    scores, ids = torch.topk(torch.softmax(torch.randn(e, generator=gen, device=DEV) * 2, 0), top)
    return {"case": dict(case), "x": torch.randn(h, generator=gen, device=DEV).half(), "ids": ids.float(), "weights": scores / scores.sum(),
            "up": [by_expert(t, 2 * f) for t in up], "down": [by_expert(t, h) for t in down],
            "mid": torch.zeros((top, 2 * f), dtype=torch.float16, device=DEV), "out": torch.zeros(h, dtype=torch.float32, device=DEV),
            "workspace": quantize.Workspace(max(quantize.moe_workspace_bytes(top, 2 * f, h, g), quantize.moe_workspace_bytes(top, h, f, g)))}


def _run_q4_experts(state):
    h, f, e, top, g = (state["case"][x] for x in ("hidden", "ff", "experts", "top", "group"))
    up, down = state["up"], state["down"]
    quantize.batched_marlin_gate_up(state["x"], up[0], up[1], state["ids"], state["mid"], up[0].numel() // e, up[1].numel() // e, 2 * f, h, top,
                                    group_size=g, workspace=state["workspace"])
    quantize.batched_marlin_down_axpy(state["mid"], down[0], down[1], state["ids"], state["weights"], state["out"], down[0].numel() // e,
                                      down[1].numel() // e, h, f, top, group_size=g, workspace=state["workspace"])
    return [state["mid"], state["out"]]


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _exact_q4_experts(case, state):
    h, f, e, top, g = (case[x] for x in ("hidden", "ff", "experts", "top", "group"))

    def matrix(pair, i, k, n):
        return _unpacked(pair[0].view(e, -1)[i], pair[1].view(e, -1)[i], k, n, g)
    chosen = [int(i) for i in state["ids"].tolist()]
    mid = torch.stack([state["x"].double() @ matrix(state["up"], i, h, 2 * f) for i in chosen])
    act = _gelu(mid[:, :f]) * mid[:, f:]
    out = sum(w * (act[j] @ matrix(state["down"], i, f, h)) for j, (i, w) in enumerate(zip(chosen, state["weights"].double())))
    return [mid, out]


# ---------------------------------------------------------------------------------------------------- 4-bit decoder --

def _prepare_q4_generate(case, seed):
    s = SIZES[case["size"]]
    cfg = generate.TransformerConfig(hidden=s["width"], num_heads=s["heads"], num_kv_heads=s["kv_heads"], head_dim=s["dim"], ffn=s["ff"],
                                     vocab=s["vocab"], layers=s["depth"]["q4"], rope_theta=THETA, max_seq=(case["context"] + case["new"] + 255) // 256 * 256)
    model = generate.Q4Model(cfg, device=DEV, seed=(seed % 9973) * 1000003)
    # token t is followed by t + 1, with a margin that rounding does not reach
    model.embed.mul_(200.0)
    model.lm_head.copy_(torch.roll(model.embed, 1, 0).mul_(0.005))
    engine = generate.QuantizedGenerationEngine(model)
    engine.prefill_random_kv(case["context"], seed=seed)
    first = int(torch.randint(0, s["vocab"] - case["new"], (1,), generator=_generator("first", seed), device=DEV))
    return {"engine": engine, "context": case["context"], "new": case["new"], "first": first}


def _run_q4_generate(state):
    engine, n0, new = state["engine"], state["context"], state["new"]
    engine.set_position(n0)
    engine.reset_history()
    tokens = engine.generate_tw_marlin_graph(state["first"], new)
    b = engine.buf
    return {"tokens": tokens_array(tokens), "logits": b.logits, "k": [t[n0:n0 + new] for t in b.k_cache], "v": [t[n0:n0 + new] for t in b.v_cache]}


def tokens_array(tokens):
    return torch.tensor(tokens, dtype=torch.int64)


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _exact_q4_generate(case, state):
    engine, cfg, n0, new = state["engine"], state["engine"].cfg, case["context"], case["new"]
    model, d, heads, groups, g = engine.model, cfg.head_dim, cfg.num_heads, cfg.num_kv_heads, cfg.group_size
    tokens = [state["first"] + i for i in range(new)]
    x = model.embed[tokens].double()
    half = d // 2
    freq = cfg.rope_theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=DEV) / d)
    angle = torch.arange(n0, n0 + new, dtype=torch.float64, device=DEV)[:, None] * freq
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(t):
        a, b = t[..., :half], t[..., half:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)
    seen = torch.arange(n0 + new, device=DEV)[None, :] <= torch.arange(n0, n0 + new, device=DEV)[:, None]
    ks, vs = [], []
    for i, w in enumerate(model.layers):
        h = _rms(x, w.attn_norm.double(), cfg.eps)
        qkv = h @ _unpacked(*w.wqkv, cfg.hidden, cfg.q_dim + 2 * cfg.kv_dim, g) + w.bqkv.double()
        q, k, v = qkv.split([cfg.q_dim, cfg.kv_dim, cfg.kv_dim], 1)
        q, k, v = turn(q.reshape(new, heads, d)), turn(k.reshape(new, groups, d)), v.reshape(new, groups, d)
        ks.append(k.reshape(new, -1))
        vs.append(v.reshape(new, -1))
        kk = torch.cat([engine.buf.k_cache[i][:n0].double().view(n0, groups, d), k]).repeat_interleave(heads // groups, 1)
        vv = torch.cat([engine.buf.v_cache[i][:n0].double().view(n0, groups, d), v]).repeat_interleave(heads // groups, 1)
        p = torch.softmax((torch.einsum("qhd,khd->hqk", q, kk) / math.sqrt(d)).masked_fill(~seen, -math.inf), -1)
        x = x + torch.einsum("hqk,khd->qhd", p, vv).reshape(new, -1) @ _unpacked(*w.wo, cfg.q_dim, cfg.hidden, g)
        gu = _rms(x, w.ffn_norm.double(), cfg.eps) @ _unpacked(*w.wgu, cfg.hidden, 2 * cfg.ffn, g)
        x = x + (torch.nn.functional.silu(gu[:, :cfg.ffn]) * gu[:, cfg.ffn:]) @ _unpacked(*w.w_down, cfg.ffn, cfg.hidden, g)
    x = _rms(x, model.final_norm.double(), cfg.eps)
    logits = torch.cat([x @ part.double().t() for part in model.lm_head.split(16384)], 1)
    picked = logits.argmax(1).tolist()
    if picked[:-1] != tokens[1:]:
        return None                                                            # the guess of the whole sequence was wrong
    return {"tokens": tokens_array(picked), "logits": logits[-1], "k": ks, "v": vs}


# ---------------------------------------------------------------------------------------- dense-weight decoders: both --

def _config(case):
    s, name = SIZES[case["size"]], case["model"]
    length = case["tokens"] + case.get("new", 0)
    if name == "bidasun":
        mixer = {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["dim"], "vdim": s["dim"], "scale": s["dim"] ** -0.5,
                 "mask": {"size": s["window"], "keep_first": s["keep"]}}
        layer = {"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": s["ff"]}}
        return {"architecture": "Bidasun", "width": s["width"], "vocab": s["vocab"], "max_positions": max(length, 64), "norm": {"eps": 1e-5},
                "layers": [layer] * s["depth"][name]}
    linear = {"type": "gla", "mixer": {"heads": s["heads"], "dim": s["dim"], "vdim": s["dim"], "tau": TAU}}
    latent = {"type": "latent_attention", "mixer": {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot"], "vdim": s["dim"], "kv_rank": s["rank"],
              "scale": (s["dim"] + s["rot"]) ** -0.5, "rot": {"base": 10000.0, "dims": s["rot"]}, "mask": {"size": s["window"]}}}
    mlp = {"kind": "moe", "expert": {"ff": s["expert_ff"]},
           "router": {"experts": s["experts"], "top": s["top"], "groups": {"count": s["groups"], "keep": s["kept"]}}}
    return {"architecture": "Zukotar", "width": s["width"], "vocab": s["vocab"], "norm": {"eps": 1e-6}, "embedding": {"scale": EMBED_SCALE},
            "layers": [dict(latent if i % 2 else linear, mlp=mlp) for i in range(s["depth"][name])]}


def _spec(case):
    config = _config(case)
    if case["model"] == "bidasun":
        return bidasun.parse_config(config)
    return zukotar.parse_config(config, lambda name: (SIZES[case["size"]]["low"], config["width"]))


def _weights(case, seed):
    """name, shape -> the tensor as a checkpoint holds it (vectors in 32 bits, matrices in the case's type); the same whenever it is asked for."""
    dt = getattr(torch, case["dtype"])

    def get(name, shape):
        leaf, gen = name.split(".")[-1], _generator(seed, "embed" if name == "head" else name)

        def normal(std):
            return torch.randn(shape, generator=gen, device=DEV).mul_(std)

        def uniform(lo, hi):
            return torch.rand(shape, generator=gen, device=DEV) * (hi - lo) + lo
        if name == "final.norm" and case["model"] == "zukotar":                 # see embed
            out = uniform(0.7, 1.3)
            out[shape[0] // 2:].neg_()
            return out
        if "norm" in leaf:
            return uniform(0.7, 1.3)
        if leaf == "pb":
            return torch.full(shape, -4.0, device=DEV)
        if leaf in ("shift", "r1", "r2"):
            return uniform(0.0, 1.0)
        if name.endswith("a2.b"):
            return uniform(0.0, 6.0)
        if name == "embed" and case["model"] == "zukotar":
            # rows in pairs that differ in the sign of their second half: with the final norm's signs, either predicts the other
            out = normal(1.0)
            out[1::2] = out[0::2]
            out[1::2, shape[1] // 2:].neg_()
            return out.to(dt)
        if name == "embed":
            return normal(2.0).to(dt)
        if name == "head":                                                      # token t is followed by t + 1
            return torch.roll(normal(2.0), 1, 0).mul_(0.01).to(dt)
        if leaf == "router":
            return normal(3.0 / math.sqrt(shape[1])).to(dt)
        return normal(0.02).to(dt)
    return get


def _following(case, token):
    return (token + 1) % SIZES[case["size"]]["vocab"] if case["model"] == "bidasun" else token ^ 1


def _tokens(case, seed):
    return torch.randint(0, SIZES[case["size"]]["vocab"] - 64, (case["tokens"],), generator=_generator("tokens", seed), device=DEV).tolist()


def _prepare_dense(case, seed):
    spec, get = _spec(case), _weights(case, seed)
    tensors = (bidasun if case["model"] == "bidasun" else zukotar).model_tensors(spec, get)
    model = dense.DenseModel(spec, tensors, getattr(torch, case["dtype"]), DEV)
    length = case["tokens"] + case.get("new", 0)
    return {"engine": DenseEngine(model, max_tokens=length, max_live=1), "tokens": _tokens(case, seed), "new": case.get("new", 0), "length": length}


def _states(engine, seq, length):
    """What the sequence leaves behind: keys and values, latents, or the recurrent state."""
    return [{name: t[seq][:length] if name.endswith("cache") else t[seq] for name, t in run.items() if name != "shift_state"}
            for run in engine.state.runs]


def _run_prompt(state):
    engine = state["engine"]
    seq = engine.open()
    logits = engine.step(seq, state["tokens"], [len(state["tokens"]) - 1])
    engine.close(seq)
    return {"logits": logits, "state": _states(engine, seq, len(state["tokens"]))}


def _run_generate(state):
    engine = state["engine"]
    seq = engine.open()
    tokens = engine.greedy(seq, state["tokens"], state["new"])
    engine.close(seq)
    return {"tokens": tokens_array(tokens), "logits": engine.logits[:1], "state": _states(engine, seq, state["length"] - 1)}


def _exact_dense(case, seed):
    spec, get = _spec(case), _weights(case, seed)
    shapes = (bidasun if case["model"] == "bidasun" else zukotar).tensor_shapes(spec)

    def weight(name):
        return get(name, shapes[name]).double()
    tokens, new = _tokens(case, seed), case.get("new", 0)
    prompt = len(tokens)
    for _ in range(new - 1):
        tokens = tokens + [_following(case, tokens[-1])]
    n, at = len(tokens), torch.tensor(tokens, device=DEV)
    x = weight("embed")[at]
    if case["model"] == "bidasun":
        x = x + weight("pos")[:n]
    else:
        x = x * EMBED_SCALE
    left = []
    for i, layer in enumerate(spec.layers):
        p = f"l{i}."
        if case["model"] == "bidasun":
            mixed, kept = _bidasun_mixer(x, layer.mixer, lambda name: weight(p + name), spec.eps)
            x = x + _rms(mixed, weight(p + "norm1"), spec.eps)
            y = (_gelu(x @ weight(p + "mlp.gate").t()) * (x @ weight(p + "mlp.up").t())) @ weight(p + "mlp.down").t()
            x = x + _rms(y, weight(p + "norm2"), spec.eps)
        else:
            mixer = _latent_mixer if isinstance(layer.mixer, dense.LatentAttentionSpec) else _linear_mixer
            mixed, kept = mixer(_rms(x, weight(p + "norm1"), spec.eps), layer.mixer, lambda name: weight(p + name), spec.eps)
            x = x + _rms(mixed, weight(p + "norm1b"), spec.eps)
            y = _experts(_rms(x, weight(p + "norm2"), spec.eps), layer.ff, lambda name: weight(p + "mlp." + name))
            x = x + _rms(y, weight(p + "norm2b"), spec.eps)
        left.append(kept)
    x = _rms(x[prompt - 1:], weight("final.norm"), spec.eps)
    logits = x @ weight("head" if case["model"] == "bidasun" else "embed").t()
    if not new:
        return {"logits": logits, "state": left}
    picked = logits.argmax(1).tolist()
    if picked[:-1] != tokens[prompt:]:
        return None                                                            # the guess of the whole sequence was wrong
    return {"tokens": tokens_array(picked), "logits": logits[-1:], "state": left}


def _bidasun_mixer(x, m, weight, eps):
    n = x.shape[0]
    h = x + (torch.cat([torch.zeros_like(x[:1]), x[:-1]]) - x) * weight("shift")
    q = _rms(h @ weight("mix.q").t(), weight("mix.q.norm"), eps).reshape(n, m.heads, m.dim)
    k = _rms(h @ weight("mix.k").t(), weight("mix.k.norm"), eps)
    v = h @ weight("mix.v").t()
    r1, r2, pb = weight("mix.r1"), weight("mix.r2"), weight("mix.pb")
    o = torch.empty((n, m.heads, m.vdim), dtype=torch.float64, device=DEV)
    dist = (torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)[None, :]).clamp_(min=0)
    seen = _seen(n, m.window, m.keep_first)
    kh, vh = k.reshape(n, m.kv_heads, m.dim), v.reshape(n, m.kv_heads, m.vdim)
    for i in range(m.heads):
        j = i * m.kv_heads // m.heads
        s = (q[:, i] @ kh[:, j].t()) * m.scale - r1[i] * torch.log1p(r2[i] * dist) + pb[i]
        o[:, i] = torch.sigmoid(s).masked_fill_(~seen, 0.0) @ vh[:, j]
    o = o.reshape(n, -1) * torch.sigmoid(h @ weight("mix.g").t())
    return o @ weight("mix.o").t(), {"k_cache": k, "v_cache": v}


def _seen(n, window, keep=0):
    i, j = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
    return (j <= i) & ((i - j < window) | (j < keep))


def _latent_mixer(h, m, weight, eps):
    n = h.shape[0]
    angle = torch.arange(n, dtype=torch.float64, device=DEV)[:, None] * m.rot_base ** (-2.0 * torch.arange(m.rot_dim // 2, dtype=torch.float64, device=DEV) / m.rot_dim)
    cos, sin = angle.cos(), angle.sin()

    def turn(t):                                                               # [n, ..., rot_dim], pairs of neighbours
        shape = (n,) + (1,) * (t.dim() - 2) + (-1,)
        c, s, a, b = cos.reshape(shape), sin.reshape(shape), t[..., 0::2], t[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    q = (h @ weight("mix.q").t()).reshape(n, m.heads, m.dim + m.rot_dim)
    q = torch.cat([q[..., :m.dim], turn(q[..., m.dim:])], -1)
    down = h @ weight("mix.dkv").t()
    latent, shared = _rms(down[:, :m.rank], weight("mix.dkv.norm"), eps), turn(down[:, m.rank:])
    k, v = (latent @ weight("mix.uk").t()).reshape(n, m.heads, m.dim), (latent @ weight("mix.uv").t()).reshape(n, m.heads, m.vdim)
    o, seen = torch.empty_like(v), _seen(n, m.window)
    for i in range(m.heads):
        s = (q[:, i] @ torch.cat([k[:, i], shared], -1).t()) * m.scale
        o[:, i] = torch.softmax(s.masked_fill_(~seen, -math.inf), -1) @ v[:, i]
    o = o * torch.sigmoid(h @ weight("mix.g").t())[:, :, None]
    return o.reshape(n, -1) @ weight("mix.o").t(), {"latent_cache": torch.cat([latent, shared], 1)}


def _linear_mixer(h, m, weight, eps):
    n = h.shape[0]
    q = (h @ weight("mix.q").t()).reshape(n, m.heads, m.dim) * m.dim ** -0.5
    k, v = (h @ weight("mix.k").t()).reshape(n, m.heads, m.dim), (h @ weight("mix.v").t()).reshape(n, m.heads, m.vdim)
    z = (h @ weight("mix.a1").t()) @ weight("mix.a2").t() + weight("mix.a2.b")
    decay = torch.sigmoid(z).pow(1.0 / m.tau).reshape(n, m.heads, m.dim)
    s, o = torch.zeros((m.heads, m.dim, m.vdim), dtype=torch.float64, device=DEV), torch.empty_like(v)
    for t in range(n):
        s.mul_(decay[t][:, :, None]).addcmul_(k[t][:, :, None], v[t][:, None, :])
        torch.matmul(q[t][:, None], s, out=o[t][:, None])
    o = _rms(o, weight("mix.norm"), eps).reshape(n, -1) * torch.nn.functional.silu(h @ weight("mix.g").t())
    return o @ weight("mix.o").t(), {"gla_state": s}


def _experts(h, ff, weight):
    score = torch.softmax(h @ weight("router").t(), -1)
    best = score.reshape(len(h), ff.groups, -1).amax(-1)
    allowed = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(ff.keep, 1).indices, True).repeat_interleave(ff.experts // ff.groups, 1)
    value, chosen = score.masked_fill(~allowed, -1.0).topk(ff.top, 1)
    out = torch.zeros_like(h)
    for e in range(ff.experts):
        rows, slot = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            y = torch.relu(h[rows] @ weight(f"e{e}.up").t()) ** 2 @ weight(f"e{e}.down").t()
            out.index_add_(0, rows, y * value[rows, slot][:, None])
    return out


# ------------------------------------------------------------------------------------------------------------ all --

_PREPARE = {"q4_layer": _prepare_q4_layer, "q4_experts": _prepare_q4_experts, "q4_generate": _prepare_q4_generate, "prompt": _prepare_dense,
            "generate": _prepare_dense}
_RUN = {"q4_layer": _run_q4_layer, "q4_experts": _run_q4_experts, "q4_generate": _run_q4_generate, "prompt": _run_prompt, "generate": _run_generate}
_EXACT = {"q4_layer": _exact_q4_layer, "q4_experts": _exact_q4_experts, "q4_generate": _exact_q4_generate}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _RUN[state["kind"]](state)


@torch.no_grad()
def exact(case, seed):
    if case["kind"] in _EXACT:
        return _EXACT[case["kind"]](case, prepare(case, seed))
    return _exact_dense(case, seed)


def _pairs(n0, n, window, keep=0):
    """Query-key pairs of the n tokens that follow n0 others."""
    return sum(min(i + 1, window) + min(max(i + 1 - window, 0), keep) for i in range(n0, n0 + n))


def work(case):
    kind = case["kind"]
    if kind == "q4_layer":
        m, g, b = case["rows"], case["group"], 4 if case["dtype"] == "float32" else 2
        shapes = _layer_shapes(case["size"])
        return {"bytes": sum(k * n // 2 + 2 * k * n // g + b * m * (k + n) for k, n in shapes), "flops": sum(2 * m * k * n for k, n in shapes)}
    if kind == "q4_experts":
        h, f, top, g = case["hidden"], case["ff"], case["top"], case["group"]
        weights = top * 3 * h * f
        return {"bytes": weights // 2 + 2 * weights // g + 2 * h + 4 * top * f + 4 * h, "flops": 2 * weights}
    s = SIZES[case["size"]]
    w, d, kv, v = s["width"], s["dim"], s["kv_heads"] * s["dim"], s["vocab"]
    q = s["heads"] * d
    if kind == "q4_generate":
        depth, new, n0 = s["depth"]["q4"], case["new"], case["context"]
        weights = depth * (w * (q + 2 * kv) + q * w + 3 * w * s["ff"])
        cache = depth * 2 * kv * sum(n0 + i + 1 for i in range(new))
        return {"bytes": new * (weights // 2 + 2 * weights // 128 + 2 * v * w) + 2 * cache,
                "flops": 2 * new * (weights + v * w) + depth * 4 * q * sum(n0 + i + 1 for i in range(new))}
    depth, b = s["depth"][case["model"]], 4 if case["dtype"] == "float32" else 2
    steps = [(0, case["tokens"])] + [(case["tokens"] + i, 1) for i in range(case.get("new", 1) - 1)]
    nbytes = flops = 0
    for n0, n in steps:
        head = v * w
        if case["model"] == "bidasun":
            weights = met = depth * (w * (2 * q + 2 * kv) + q * w + 3 * w * s["ff"])
            mix = depth * 4 * q * _pairs(n0, n, s["window"], s["keep"])
            state = depth * 2 * kv * (n + min(n0, s["window"] + s["keep"])) * b
        else:
            linear = w * (4 * q + s["low"]) + q * s["low"] + q * w
            latent = w * (s["heads"] * (d + s["rot"]) + s["rank"] + s["rot"] + s["heads"]) + s["rank"] * 2 * q + q * w
            expert, e = 2 * w * s["expert_ff"], s["experts"]
            touched = e * (1.0 - (1.0 - s["top"] / e) ** n)                     # experts that n tokens meet, evenly dealt
            mixers = depth // 2 * (linear + latent) + depth * e * w
            weights, met = mixers + depth * touched * expert, mixers + depth * s["top"] * expert
            # scores and values over what a query sees; a recurrence step moves and reads a matrix per head
            mix = depth // 2 * (2 * s["heads"] * (2 * d + s["rot"]) * _pairs(n0, n, s["window"]) + 4 * n * q * d)
            state = depth // 2 * ((s["rank"] + s["rot"]) * (n + min(n0, s["window"])) * b + (2 if n0 else 1) * 4 * q * d)
        nbytes += b * (weights + head) + state + 4 * v
        flops += 2 * n * met + mix + 2 * head
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """About four times what the path differs from ``exact`` by (given in front of each)."""
    if case["kind"] in ("q4_layer", "q4_experts"):
        return {"rel": 2e-6} if case.get("dtype") == "float32" else {"rel": 1.5e-3}       # 4e-7; 2e-4 to 4e-4
    if case["kind"] == "q4_generate":
        return {"rel": 6e-3}                                                               # 1.5e-3
    if case["dtype"] == "float32":
        return {"rel": 2e-5}                                                               # 4e-6
    return {"rel": 0.03, "max": 0.99}                                                      # 6e-3 to 9e-3; to 1.4e-2 and 0.4 where experts are chosen
