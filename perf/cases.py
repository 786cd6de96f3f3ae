"""What a user of this library has it do, as cases that can be timed and checked.

Most cases are one batch of requests through `Model.open`, `Model.step` and `Model.close`: the prompts of all
sequences go in one step, then every sequence brings one token a step for `steps` steps, and the slots are given
back.  The tokens that follow the prompts are given (as in trace replay), so that the outputs, the logits of every
step, do not hang on near-ties.  `steps` 0 is a pure prompt.  The rest choose tokens from logits with `Sampler`.

Sizes are those that bench.py measures: the dense decoder at its presets, and one decoder of each kind of mixer
(latent attention with experts; windowed attention beside gated linear attention, and state-space layers; residual
streams with lightning layers and experts; a delta rule beside convolved and low-rank attention) at widths 1024 to
4096.  Weights are random with the distributions of the random-weights mode, but for three: the experts' routers are
three times as wide, because a trained router tells its experts apart; and the dense decoder, which runs at its full
depth too, has embeddings of unit size and, as deep decoders are initialised, output and down projections divided by
sqrt(2 layers), so that bfloat16 rounding does not pile up over its layers as no trained network lets it.

`exact` computes the same logits in 64 bits with plain torch, whole sequences at a time, from the equations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from braidinfer_b200 import Model, SamplingParams
from braidinfer_b200.config import preset
from braidinfer_b200.engine import Engine
from braidinfer_b200.models import architecture_for
from braidinfer_b200.weights import tensor_specs_of

DEVICE = "cuda:0"
D = torch.float64
VOCAB = 32768
PAGE = 64

# ------------------------------------------------------------------------------------------------ configurations
HYBRID = {   # width, attention heads / kv heads / head size / window, recurrent heads / key / value size, state-space sizes, ff, side
    "w1024": dict(width=1024, heads=8, kv=2, dim=64, window=512, lheads=4, ldk=64, ldv=128, sheads=32, sp=64, sn=64, sg=4, ff=2816, side=128),
    "w2048": dict(width=2048, heads=16, kv=4, dim=128, window=1024, lheads=8, ldk=128, ldv=256, sheads=64, sp=64, sn=128, sg=8, ff=5632,
                  side=256),
    "w4096": dict(width=4096, heads=32, kv=8, dim=128, window=1024, lheads=16, ldk=128, ldv=256, sheads=128, sp=64, sn=128, sg=8, ff=14336,
                  side=256),
}
LATENT = {   # heads, unrotated / rotated / value size a head, ranks of queries and keys, inner size of the delta layers' gates
    "w1024": dict(heads=8, dim=64, rot=32, vdim=64, q_rank=512, kv_rank=256, low=64),
    "w2048": dict(heads=16, dim=128, rot=64, vdim=128, q_rank=1024, kv_rank=512, low=128),
    "w4096": dict(heads=32, dim=128, rot=64, vdim=128, q_rank=1536, kv_rank=512, low=128),
}
EXPERTS = {  # experts, groups, groups kept, experts a token, an expert's width
    "w1024": dict(experts=16, groups=1, keep=1, top=2, ff=1024),
    "w2048": dict(experts=64, groups=8, keep=4, top=6, ff=1408),
    "w4096": dict(experts=32, groups=4, keep=2, top=4, ff=2048),
}
DENSE = {    # the dense decoder at four layers: width, heads, kv heads, head size, ff
    "w1024": dict(width=1024, heads=8, kv=2, dim=64, ff=2816),
    "w2048": dict(width=2048, heads=16, kv=4, dim=128, ff=5632),
    "w4096": dict(width=4096, heads=32, kv=8, dim=128, ff=14336),
}


def config(model, size):
    """config.json of a model: what a model folder would hold."""
    if model == "dense":
        if size not in DENSE:
            return preset(size)
        z = DENSE[size]
        return {"architectures": ["MistralForCausalLM"], "model_type": "mistral", "torch_dtype": "bfloat16", "num_hidden_layers": 4,
                "hidden_size": z["width"], "num_attention_heads": z["heads"], "num_key_value_heads": z["kv"], "head_dim": z["dim"],
                "intermediate_size": z["ff"], "vocab_size": VOCAB, "rope_theta": 1e6, "rms_norm_eps": 1e-5, "sliding_window": None,
                "tie_word_embeddings": False, "max_position_embeddings": 32768}
    z, y, x = HYBRID[size], LATENT[size], EXPERTS[size]
    width = z["width"]
    if model == "bidinex":
        mixer = {"heads": y["heads"], "dim": y["dim"], "rot_dim": y["rot"], "rot": {"base": 10000.0, "dims": y["rot"]}, "vdim": y["vdim"],
                 "kv_rank": y["kv_rank"], "scale": (y["dim"] + y["rot"]) ** -0.5}
        mlp = {"kind": "moe", "expert": {"ff": x["ff"]},
               "router": {"experts": x["experts"], "top": x["top"], "groups": {"count": x["groups"], "keep": x["keep"]}}}
        return {"architecture": "Bidinex", "vocab": VOCAB, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
                "residual_mult": 1.0, "logit_softcap": 30.0, "loop": None,
                "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp} for _ in range(4)]}
    ff = {"kind": "dense", "ff": z["ff"]}
    heads = {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["dim"], "scale": z["dim"] ** -0.5,
             "mask": {"size": z["window"]}}
    if model == "loduzen":
        left = dict(heads, rot={"base": 1e6, "dims": z["dim"] // 2, "scaling": {"factor": 4.0, "original": 4096, "fast": 16.0, "slow": 2.0}})
        right = {"heads": z["lheads"], "dim": z["ldk"], "vdim": z["ldv"], "tau": 8.0}
        par = {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}, "mlp": ff}
        ssm = {"type": "mamba2", "mixer": {"heads": z["sheads"], "vdim": z["sp"], "state": z["sn"], "groups": z["sg"], "conv": 4,
                                           "norm_groups": z["sg"]}, "mlp": ff}
        return {"architecture": "Loduzen", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "token_side": {"dim": z["side"]},
                "layers": [par, ssm, par, ssm]}
    if model == "zisesun":
        mem = {"heads": z["lheads"], "dim": z["ldk"], "vdim": z["ldv"], "decay": [1.0 - 2.0 ** -(3 + h) for h in range(z["lheads"])]}
        moe = {"kind": "moe", "expert": {"ff": z["ff"] // 2 // 64 * 64}, "router": {"experts": 8, "top": 2}}
        att, lit = {"type": "attention", "mixer": heads, "mlp": moe}, {"type": "lightning", "mixer": mem, "mlp": moe}
        return {"architecture": "Zisesun", "vocab": VOCAB, "width": width, "streams": 4, "max_positions": 16384, "norm": {"eps": 1e-6},
                "layers": [att, lit, att, lit]}
    if model == "megerax":
        att = dict(heads, conv=4, softcap=50.0,
                   rot={"base": 1e6, "dims": z["dim"] // 2, "scaling": {"factor": 4.0, "low": 1.0, "high": 4.0, "original": 4096}})
        delta = {"heads": z["lheads"], "kv_heads": z["lheads"], "dim": z["ldk"], "vdim": z["ldv"], "conv": 4, "decay_rank": y["low"],
                 "gate_rank": y["low"]}
        lat = {"heads": y["heads"], "dim": y["dim"], "rot_dim": y["rot"], "vdim": y["vdim"], "q_rank": y["q_rank"], "kv_rank": y["kv_rank"],
               "scale": (y["dim"] + y["rot"]) ** -0.5, "rot": {"base": 1e6, "dims": y["rot"]}}
        d = {"type": "channel_delta", "mixer": delta, "mlp": None}
        return {"architecture": "Megerax", "vocab": VOCAB, "width": width, "logit_scale": 0.5, "norm": {"eps": 1e-6},
                "layers": [{"type": "latent_attention", "mixer": lat, "mlp": ff}, d, {"type": "attention", "mixer": att, "mlp": ff}, d]}
    raise ValueError(model)


# ------------------------------------------------------------------------------------------------ cases
def _turn(model, size, seqs, longest, steps, dtype="bfloat16", **kw):
    return dict(kw, do="turn", model=model, size=size, seqs=seqs, longest=longest, steps=steps, dtype=dtype)


def _sample(rows, vocab, temperature, top_k, top_p, **kw):
    return dict(kw, do="sample", rows=rows, vocab=vocab, temperature=temperature, top_k=top_k, top_p=top_p)


def listed():
    return [
        # one user and a short question to a 7B model: launches and latency of a batch of one
        _turn("dense", "mistral_7b_v03", 1, 37, 16, name="dense_one"),
        # the headline: eight requests of unequal length, mostly decoding
        _turn("dense", "mistral_7b_v03", 8, 512, 32, name="dense_eight"),
        # a long document's prompt
        _turn("dense", "mistral_7b_v03", 1, 2048, 0, name="dense_prompt"),
        # the true 32-bit path, as used to check a conversion
        _turn("dense", "w1024", 3, 200, 8, "float32", name="dense_float32"),
        # latent attention and experts: a long prompt, then a batch that decodes
        _turn("bidinex", "w2048", 1, 2048, 0, name="bidinex_prompt"),
        _turn("bidinex", "w2048", 8, 256, 24, name="bidinex_decode"),
        # attention beside recurrences: three unequal prompts, then a small model's batch that decodes
        _turn("loduzen", "w2048", 3, 1500, 0, name="loduzen_prompts"),
        _turn("loduzen", "w1024", 8, 61, 24, name="loduzen_decode"),
        # residual streams, lightning layers and experts: both directions in one turn
        _turn("zisesun", "w2048", 4, 700, 12, name="zisesun_turn"),
        # a delta rule beside low-rank attention: unequal prompts of a wide model, and a few sequences that decode
        _turn("megerax", "w4096", 2, 1777, 0, name="megerax_prompts"),
        _turn("megerax", "w2048", 5, 130, 24, name="megerax_decode"),
        # choosing the tokens of a batch with the default options
        _sample(64, VOCAB, 1.0, 50, 1.0, name="sample"),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.1:
        return _sample(_between(rng, 1, 64), rng.choice([32000, VOCAB, 50257]), rng.choice([0.0, 0.7, 1.0]), rng.choice([0, 20, 50]),
                       rng.choice([0.9, 1.0]))
    model = rng.choice(["dense", "bidinex", "loduzen", "zisesun", "megerax"])
    size = rng.choice(["w1024", "w2048", "w4096"] + (["mistral_7b_v03"] if model == "dense" else []))
    dtype = "float32" if size == "w1024" and rng.random() < 0.2 else "bfloat16"
    seqs = _between(rng, 1, 16)
    most = 2300 if size == "mistral_7b_v03" else 600 if dtype == "float32" else 4096
    longest = min(_between(rng, 5, 2500), most // seqs)
    steps = 0 if rng.random() < 0.4 else _between(rng, 2, 24)
    return _turn(model, size, seqs, longest, steps, dtype)


def lengths(case):
    """The prompts' lengths: the longest, and ever shorter ones down to about two fifths of it."""
    n = case["seqs"]
    return [max(1, round(case["longest"] * (1 - 0.6 * i / n))) for i in range(n)]


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _specs(cfg):
    arch = architecture_for(cfg)
    return tensor_specs_of(arch.build_spec(arch.config_from_dict(cfg)))


def _factor(cfg, name):
    if name.endswith(".router"):
        return 3.0
    if name == "model.embed_tokens.weight":
        return 50.0
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        return (2 * cfg["num_hidden_layers"]) ** -0.5
    return 1.0


def weights(case, seed):
    cfg, g, out = config(case["model"], case["size"]), _generator(seed), {}
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    for name, ts in _specs(cfg).items():
        x = torch.empty(ts.shape, dtype=dtype, device=DEVICE).normal_(0.0, ts.std * _factor(cfg, name), generator=g)
        if ts.init == "one_plus_normal":
            x += 1.0
        elif ts.init == "eye_plus_normal":
            x += torch.eye(ts.shape[0], dtype=dtype, device=DEVICE)
        out[name] = x
    return out


def tokens(case, seed):
    """(prompts, the tokens that each sequence brings after its prompt)."""
    rng = np.random.RandomState(seed % (1 << 31))
    return ([rng.randint(0, VOCAB, n).tolist() for n in lengths(case)],
            [rng.randint(0, VOCAB, case["steps"]).tolist() for _ in range(case["seqs"])])


def sample_logits(case, seed):
    """Rows with a few likely tokens over a long tail."""
    g = _generator(seed)
    x = torch.randn(case["rows"], case["vocab"], device=DEVICE, generator=g) * 2.0
    return x + 4.0 * torch.rand(case["rows"], case["vocab"], device=DEVICE, generator=g).pow(64)


def prepare(case, seed):
    if case["do"] == "sample":
        # a small model's sampler: choosing tokens does not depend on the model
        eng = Engine.from_random(preset("tiny_a"), 0, max_tokens=PAGE, max_slots=1, verbose=False)
        p = SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"])
        rows = list(range(case["rows"]))
        return {"do": "sample", "sampler": Model(eng, 1).sampler, "logits": sample_logits(case, seed), "params": [p] * len(rows),
                "seeds": [int(seed) + r for r in rows], "ids": rows, "at": [0] * len(rows)}
    room = sum(-(-(n + case["steps"]) // PAGE) * PAGE for n in lengths(case))
    eng = Engine(config(case["model"], case["size"]), weights(case, seed), dtype=case["dtype"], max_tokens=room, max_slots=case["seqs"],
                 device=DEVICE, verbose=False)
    prompts, follow = tokens(case, seed)
    return {"do": "turn", "model": Model(eng, case["seqs"]), "prompts": prompts, "follow": follow, "steps": case["steps"]}


def run(state):
    if state["do"] == "sample":
        s = state
        return np.asarray(s["sampler"].choose(s["logits"], s["params"], s["seeds"], s["ids"], s["at"]))
    model, follow = state["model"], state["follow"]
    slots = [model.open() for _ in state["prompts"]]
    out = [model.step(list(zip(slots, state["prompts"])))]
    steps = [model.step([(s, [f[t]]) for s, f in zip(slots, follow)]) for t in range(state["steps"])]
    for s in slots:
        model.close(s)
    return out + [torch.cat(steps)] if steps else out


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Every step reads the weights that its tokens use once, and the keys, values or states of its sequences; a prompt's
    products and attention are counted once a token, the recurrences as one walk."""
    if case["do"] == "sample":
        return {"bytes": case["rows"] * (case["vocab"] * 4 + 4), "flops": 0}
    cfg = config(case["model"], case["size"])
    size = 4 if case["dtype"] == "float32" else 2
    plain = expert = 0
    table = cfg.get("vocab", cfg.get("vocab_size")) * cfg.get("width", cfg.get("hidden_size"))
    for name, ts in _specs(cfg).items():
        n = math.prod(ts.shape)
        if ".mlp.e" in name:
            expert += n
        elif "embed" not in name and "head" not in name and not name.endswith("pos"):
            plain += n
    top, count = (2, 8) if case["model"] == "zisesun" else (EXPERTS[case["size"]]["top"], EXPERTS[case["size"]]["experts"]) \
        if case["model"] == "bidinex" else (0, 1)
    pair, row, state = 0, 0, 0            # FLOPs of a query and key, numbers a cached token, 32-bit numbers of state a sequence
    window = None
    if case["model"] == "dense":
        L = cfg["num_hidden_layers"]
        pair, row = L * 4 * cfg["num_attention_heads"] * cfg["head_dim"], L * 2 * cfg["num_key_value_heads"] * cfg["head_dim"]
    else:
        z, y = HYBRID[case["size"]], LATENT[case["size"]]
        lat_pair, lat_row = 2 * y["heads"] * (y["dim"] + y["rot"] + y["vdim"]), y["kv_rank"] + y["rot"]
        att_pair, att_row, mem = 4 * z["heads"] * z["dim"], 2 * z["kv"] * z["dim"], z["lheads"] * z["ldk"] * z["ldv"]
        if case["model"] == "bidinex":
            pair, row = 4 * lat_pair, 4 * lat_row
        elif case["model"] == "megerax":
            pair, row, state = lat_pair + att_pair, lat_row + att_row, 2 * mem
        else:
            pair, row, window = 2 * att_pair, 2 * att_row, z["window"]
            state = 2 * mem + (2 * z["sheads"] * z["sp"] * z["sn"] if case["model"] == "loduzen" else 0)

    def seen(n):
        return min(n, window) if window else n

    nbytes = flops = 0
    ls = lengths(case)
    for t in range(case["steps"] + 1):
        new = sum(ls) if t == 0 else len(ls)
        touched = expert * (1 - (1 - top / count) ** new)
        nbytes += (plain + touched + table) * size + len(ls) * VOCAB * 4
        flops += 2 * (plain + expert * top / count) * new + 2 * table * len(ls) + 4 * state * new
        for n in ls:
            if t == 0:
                pairs = sum(seen(i + 1) for i in range(n))
                nbytes += n * row * size + state * 4
            else:
                pairs = seen(n + t)
                nbytes += (pairs + 1) * row * size + 2 * state * 4
            flops += pairs * pair
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Measured between runs with other orders of sums and other kernels, and stated at about four times that (bfloat16
    between the kernels of a layer, over 4 or 32 layers: 0.002 to 0.015; 32-bit sums in the float32 runs: 3e-6 beside `exact`)."""
    if case["do"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5, "max": 3e-4}
    return {"rel": 0.03, "max": 0.6}


# ------------------------------------------------------------------------------------------------ 64 bits
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _rotate(x, freq, halves, amplitude=1.0):
    """x [T, heads, n]: the first 2 len(freq) numbers of a head turn by position * freq; pairs are neighbours, or
    numbers half of that apart."""
    n = 2 * freq.numel()
    a = torch.arange(x.shape[0], dtype=D, device=x.device)[:, None, None] * freq
    c, s = torch.cos(a) * amplitude, torch.sin(a) * amplitude
    out = x.clone()
    first, second = (slice(0, n // 2), slice(n // 2, n)) if halves else (slice(0, n, 2), slice(1, n, 2))
    u, v = x[..., first], x[..., second]
    out[..., first], out[..., second] = u * c - v * s, v * c + u * s
    return out


def _plain_freq(base, n):
    return base ** (-2.0 * torch.arange(n // 2, dtype=D, device=DEVICE) / n)


def _attend(q, k, v, change, window=None, sink=None):
    """q [T, H, .], k [T, G, .], v [T, G, .]; `change(scores, head, distance)`; `sink` joins the denominator."""
    T, H = q.shape[:2]
    per = H // k.shape[1]
    dist = torch.arange(T, device=q.device)[:, None] - torch.arange(T, device=q.device)[None]
    hidden = dist < 0
    if window:
        hidden = hidden | (dist >= window)
    out = torch.empty(T, H, v.shape[-1], dtype=D, device=q.device)
    for h in range(H):
        s = change(q[:, h] @ k[:, h // per].T, h, dist).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].reshape(1, 1).expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, h // per]
    return out.reshape(T, -1)


def _scan(decay, k, v, q):
    """S <- decay S + k v^T, o = S^T q, token by token; decay [T, H, dk], k and q [T, H, dk], v [T, H, dv]."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=D, device=k.device)
    out = torch.empty_like(v)
    for t in range(k.shape[0]):
        S.mul_(decay[t][:, :, None]).baddbmm_(k[t][:, :, None], v[t][:, None, :])
        torch.bmm(q[t][:, None, :], S, out=out[t][:, None, :])
    return out


def _conv(x, w, b=None):
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _chosen_experts(h, w, idx, share, count):
    out = torch.zeros_like(h)
    for e in range(count):
        rows, at = (idx == e).nonzero(as_tuple=True)
        if rows.numel():
            x = h[rows]
            y = (_silu(x @ w(f"e{e}.gate").T) * (x @ w(f"e{e}.up").T)) @ w(f"e{e}.down").T
            out.index_add_(0, rows, y * share[rows, at][:, None])
    return out


def _latent(h, w, q, m, change, sink=None):
    """Keys and values through a low-rank vector, one rotated key part for all heads; q [T, heads, dim + rot_dim]."""
    T, H, d, r = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    f = _plain_freq(m["rot"]["base"], m["rot"]["dims"])
    z = h @ w("dkv").T
    c = _unit(z[:, :r], m["eps"]) * w("dkv.norm")
    kr = _rotate(z[:, None, r:], f, True).expand(T, H, -1)
    k = torch.cat([(c @ w("uk").T).view(T, H, d), kr], -1)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], f, True)], -1)
    return _attend(q, k, (c @ w("uv").T).view(T, H, m["vdim"]), change, None, sink)


def _scaled(scale):
    return lambda s, h, dist: s * scale


def _dense_model(cfg, w, toks):
    H, G, d, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    x = w("model.embed_tokens.weight", toks)
    f = _plain_freq(cfg["rope_theta"], d)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _unit(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).view(len(toks), -1, d) for n in "qkv")
        x = x + _attend(_rotate(q, f, True), _rotate(k, f, True), v, _scaled(d ** -0.5), cfg["sliding_window"]) \
            @ w(p + "self_attn.o_proj.weight").T
        h = _unit(x, eps) * w(p + "post_attention_layernorm.weight")
        x = x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    return lambda rows: (_unit(x[rows], eps) * w("model.norm.weight")) @ w("lm_head.weight").T


def _bidinex(cfg, w, toks):
    def dyt(x, n):
        return torch.tanh(w(n + ".alpha") * x) * w(n) + w(n + ".b")

    x = dyt(w("embed", toks), "embed.norm")
    for i, L in enumerate(cfg["layers"]):
        m, g = dict(L["mixer"], eps=cfg["norm"]["eps"]), L["mlp"]["router"]
        mix, mlp = (lambda n, p=f"l{i}.mix.": w(p + n)), (lambda n, p=f"l{i}.mlp.": w(p + n))
        h = dyt(x, f"l{i}.norm1")
        y = _latent(h, mix, (h @ mix("q").T).view(len(toks), m["heads"], -1), m, _scaled(m["scale"]))
        y = (y.view(len(toks), m["heads"], -1) * torch.sigmoid(h @ mix("g").T)[:, :, None]).reshape(len(toks), -1)
        x = x + y @ mix("o").T
        h = dyt(x, f"l{i}.norm2")
        s = torch.softmax(h @ mlp("router").T, -1)
        best = s.view(len(toks), g["groups"]["count"], -1).max(-1).values.topk(g["groups"]["keep"], -1).indices
        kept = torch.zeros(len(toks), g["groups"]["count"], dtype=torch.bool, device=x.device).scatter_(1, best, True)
        allowed = s.masked_fill(~kept.repeat_interleave(g["experts"] // g["groups"]["count"], 1), -1.0)
        share, idx = allowed.topk(g["top"], -1)
        x = x + _chosen_experts(h, mlp, idx, share / share.sum(-1, keepdim=True), g["experts"])
    cap = cfg["logit_softcap"]
    return lambda rows: cap * torch.tanh(dyt(x[rows], "final.norm") @ w("embed").T / cap)


def _loduzen(cfg, w, toks):
    T, eps, side = len(toks), cfg["norm"]["eps"], cfg["token_side"]["dim"]
    x = w("embed", toks)
    for i, L in enumerate(cfg["layers"]):
        h = _unit(x, eps) * w(f"l{i}.norm1")
        if L["type"] == "parallel":
            m, lw = L["mixer"]["left"], (lambda n, p=f"l{i}.mix.left.": w(p + n))
            n, base, sc = m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]
            at = torch.arange(n // 2, dtype=D, device=x.device)
            lo, hi = (n * math.log(sc["original"] / (2 * math.pi * sc[t])) / (2 * math.log(base)) for t in ("fast", "slow"))
            lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), n - 1)
            ramp = ((at - lo) / max(hi - lo, 0.001)).clamp(0, 1)
            f, amp = _plain_freq(base, n) * (ramp / sc["factor"] + 1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
            q, k = (h @ lw("q").T).view(T, -1, m["dim"]), (h @ lw("k").T).view(T, -1, m["dim"])
            y = _attend(_rotate(_unit(q, eps) * lw("q.norm"), f, False, amp), _rotate(_unit(k, eps) * lw("k.norm"), f, False, amp), k,
                        _scaled(m["scale"]), m["mask"]["size"], torch.zeros(m["heads"], dtype=D, device=x.device)) @ lw("o").T
            r, rw = L["mixer"]["right"], (lambda n, p=f"l{i}.mix.right.": w(p + n))
            q, k, v = ((h @ rw(n).T).view(T, r["heads"], -1) for n in "qkv")
            decay = torch.sigmoid((h @ rw("a1").T) @ rw("a2").T + rw("a2.b")).pow(1.0 / r["tau"]).view(T, r["heads"], -1)
            o = _unit(_scan(decay, k, v, q * r["dim"] ** -0.5), eps) * rw("norm")
            y = L["mixer"]["left_scale"] * y + L["mixer"]["right_scale"] * ((o.reshape(T, -1) * _silu(h @ rw("g").T)) @ rw("o").T)
        else:
            m, mw = L["mixer"], (lambda n, p=f"l{i}.mix.": w(p + n))
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            z, ubc, dt = (h @ mw("in").T).split([H * P, H * P + 2 * G * N, H], -1)
            u, B, C = _silu(_conv(ubc, mw("conv"), mw("conv.b"))).split([H * P, G * N, G * N], -1)
            u, B, C = u.view(T, H, P), *(t.view(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
            dt = torch.nn.functional.softplus(dt + mw("dt_bias"))
            decay = torch.exp(-torch.exp(mw("A_log")) * dt)[:, :, None].expand(T, H, N)
            y = _scan(decay, B * dt[:, :, None], u, C) + mw("D")[:, None] * u
            y = (y.reshape(T, -1) * _silu(z)).view(T, m["norm_groups"], -1)
            y = (_unit(y, eps).reshape(T, -1) * mw("norm")) @ mw("o").T
        x = x + y
        h, p = _unit(x, eps) * w(f"l{i}.norm2"), f"l{i}.mlp."
        x = x + (_gelu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T
        e, p = w("side.embed", toks)[:, i * side:(i + 1) * side], f"l{i}.side."
        x = x + _unit((_gelu(x @ w(p + "gate").T) * e) @ w(p + "proj").T, eps) * w(p + "norm")
    return lambda rows: (_unit(x[rows], eps) * w("final.norm")) @ w("embed").T


def _zisesun(cfg, w, toks):
    T, eps = len(toks), cfg["norm"]["eps"]
    X = (w("embed", toks) + w("pos", range(T)))[None].repeat(cfg["streams"], 1, 1)

    def attention(h, mw, m):
        q = (_unit(h @ mw("q").T + mw("q.b"), eps) * mw("q.norm")).view(T, -1, m["dim"])
        k = (_unit(h @ mw("k").T + mw("k.b"), eps) * mw("k.norm")).view(T, -1, m["dim"])
        v = _unit((h @ mw("v").T + mw("v.b")).view(T, -1, m["vdim"]), eps)
        r1, r2 = mw("r1"), mw("r2")
        return _attend(q, k, v, lambda s, a, d: s * m["scale"] - r1[a] * torch.log(1.0 + r2[a] * d.clamp_min(0).to(D)),
                       m["mask"]["size"]) @ mw("o").T

    def lightning(h, mw, m):
        q, k, v = (_silu(h @ mw(n).T).view(T, m["heads"], -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=D, device=h.device)[None, :, None].expand(T, -1, m["dim"])
        y = _unit(_scan(decay, k, v, q).reshape(T, -1), eps) * mw("norm")
        return (y * torch.sigmoid(h @ mw("g").T)) @ mw("o").T

    def experts(h, mw, m):
        s = torch.softmax(h @ mw("router").T, -1)
        idx = (s + mw("correction")).topk(m["router"]["top"], -1).indices
        return _chosen_experts(h, mw, idx, s.gather(-1, idx), m["router"]["experts"])

    for i, L in enumerate(cfg["layers"]):
        for n, part, p, m in ((1, attention if L["type"] == "attention" else lightning, "mix.", L["mixer"]), (2, experts, "mlp.", L["mlp"])):
            hc = f"l{i}.hc{n}."
            u = torch.einsum("s,stw->tw", w(hc + "in"), X)
            y = part(_unit(u, eps) * w(f"l{i}.norm{n}"), lambda t, p=f"l{i}.{p}": w(p + t), m)
            X = torch.einsum("sr,stw->rtw", w(hc + "mix"), X) + w(hc + "out")[:, None, None] * y
    return lambda rows: (_unit(X.sum(0)[rows], eps) * w("final.norm")) @ w("head").T


def _megerax(cfg, w, toks):
    T, eps = len(toks), cfg["norm"]["eps"]

    def latent(h, mw, m):
        q = ((_unit(h @ mw("dq").T, eps) * mw("dq.norm")) @ mw("uq").T).view(T, m["heads"], -1)
        return _latent(h, mw, q, dict(m, eps=eps), _scaled(m["scale"]), mw("sink")) @ mw("o").T

    def attention(h, mw, m):
        sc, f = m["rot"]["scaling"], _plain_freq(m["rot"]["base"], m["rot"]["dims"])
        turns = sc["original"] * f / (2 * math.pi)
        keep = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        f = f * (keep + (1 - keep) / sc["factor"])
        q, k, v = (_conv(h @ mw(n).T + mw(n + ".b"), mw(n + ".conv")).view(T, -1, m["dim"]) for n in "qkv")
        q, k = (_rotate(_unit(t, eps) * mw(n + ".norm"), f, False) for n, t in (("q", q), ("k", k)))
        cap = m["softcap"]
        y = _attend(q, k, v, lambda s, a, d: cap * torch.tanh(s * m["scale"] / cap), m["mask"]["size"])
        return (y * torch.sigmoid(h @ mw("g").T)) @ mw("o").T

    def delta(h, mw, m):
        H, dk = m["heads"], m["dim"]
        q, k, v = (_silu(_conv(h @ mw(n).T, mw(n + ".conv"))).view(T, H, -1) for n in "qkv")
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q = q * dk ** -0.5
        z = torch.nn.functional.softplus((h @ mw("a1").T) @ mw("a2").T + mw("dt_bias")).view(T, H, dk)
        g = torch.exp(-torch.exp(mw("A_log"))[None, :, None] * z)
        beta = torch.sigmoid(h @ mw("b").T)
        S = torch.zeros(H, dk, v.shape[2], dtype=D, device=h.device)
        o = torch.empty_like(v)
        for t in range(T):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
        gate = torch.sigmoid((h @ mw("g1").T) @ mw("g2").T)
        return ((_unit(o, eps) * mw("norm")).reshape(T, -1) * gate) @ mw("o").T

    x = _unit(w("embed", toks), eps) * w("embed.norm")
    for i, L in enumerate(cfg["layers"]):
        part = {"latent_attention": latent, "attention": attention, "channel_delta": delta}[L["type"]]
        x = x + part(_unit(x, eps) * w(f"l{i}.norm1"), lambda n, p=f"l{i}.mix.": w(p + n), L["mixer"])
        if L["mlp"] is not None:
            h, p = _unit(x, eps) * w(f"l{i}.norm2"), f"l{i}.mlp."
            x = x + (_gelu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T
    return lambda rows: cfg["logit_scale"] * ((_unit(x[rows], eps) * w("final.norm")) @ w("head").T)


_MODELS = {"dense": _dense_model, "bidinex": _bidinex, "loduzen": _loduzen, "zisesun": _zisesun, "megerax": _megerax}


def exact(case, seed):
    if case["do"] == "sample":
        return None                       # whole numbers: they are the same or they are not
    if sum(lengths(case)) > 3000 and case["model"] in ("loduzen", "zisesun", "megerax"):
        return None                       # token by token, over 20 seconds
    stored = weights(case, seed)

    def w(name, rows=None):
        t = stored[name]
        return (t if rows is None else t[torch.as_tensor(list(rows), device=t.device)]).to(D)

    cfg, per_seq = config(case["model"], case["size"]), []
    for prompt, follow in zip(*tokens(case, seed)):
        logits_of = _MODELS[case["model"]](cfg, w, prompt + follow)
        per_seq.append(logits_of(slice(len(prompt) - 1, None)))
    steps = [torch.stack([s[t] for s in per_seq]) for t in range(case["steps"] + 1)]
    return steps[:1] + [torch.cat(steps[1:])] if case["steps"] else steps
