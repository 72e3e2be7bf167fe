"""What is timed when this library's speed is followed from one state of the code to the next.

A case is a model (a design, a width, some of its layers, a compute dtype) and a step through the engine:

  prompt   `Engine.open`, `Engine.step` with whole prompts, `Engine.close`: the time to a request's first token.  Logits
           are wanted at every 128th position and at every prompt's last one.
  decode   `Engine.decode_launch`: one token for each of the sequences that live in the cache (their prompts went
           through the step function before), the captured step that generation and replay run.

The configurations are the presets', cut to fewer layers where a whole model says nothing more (one or two cases are
whole models).  The Llama decoder, which the library is about, has half of the cases: both phases, both dtypes, its
three widths, one sequence to 64.  The other designs' layers stand for those that share their mixers: state-space layers and
window attention beside a time mix (Sagizen), the delta rule, latent and chunked attention (Vosulorn), the recurrent unit
and two-map attention over four residual streams (Redenex), softmax attention beside linear attention (Radupel).
Layers here have dense feed-forwards or none: which experts a mixture picks can change with the last bit of a
sum, so its outputs cannot be compared within a tolerance.
"""
import copy
import math

import torch

from edgelm_b200.config import config_class_for
from edgelm_b200.engine.engine import Engine, StepEntry
from edgelm_b200.engine.model import DecoderModel
from edgelm_b200.presets import PRESETS
from edgelm_b200.sampling import SamplingParams

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
DEVICE = "cuda:0"
MAX_POSITIONS = 8192
WANT_EVERY = 128

# the layers of each design's preset that the cases run (None: as many as the case says, all are alike)
DESIGN_LAYERS = {"sagizen": (2, 3), "vosulorn": (0, 1, 3), "redenex": (0, 2), "radupel": (0,)}
GREEDY = SamplingParams(0.0, 40, 0)


# ----------------------------------------------------------------------------- the cases
def _case(name, preset, phase, seqs, shortest, longest, dtype="bfloat16", layers=0):
    """`layers`: of a Llama preset, how many (0: the design's list, or all)."""
    return {"name": name, "preset": preset, "phase": phase, "seqs": seqs, "shortest": shortest, "longest": longest,
            "dtype": dtype, "layers": layers}


def listed():
    return [
        # a person waits for one answer: the whole small model, one token at a time, every kernel a few microseconds
        _case("decode_135m_one", "smollm2-135m", "decode", 1, 700, 700),
        # a handful of requests on the middle size, contexts of all lengths
        _case("decode_360m_batch", "smollm2-360m", "decode", 8, 130, 2040, layers=8),
        # a full server: 64 requests on the wide model
        _case("decode_1p7b_many", "smollm2-1.7b", "decode", 64, 128, 2300, layers=4),
        # a long prompt on the small model, whole
        _case("prompt_135m_2048", "smollm2-135m", "prompt", 1, 2048, 2048),
        # requests that start together with unequal prompts on the wide model
        _case("prompt_1p7b_ragged", "smollm2-1.7b", "prompt", 7, 65, 1901, layers=2),
        # the true 32-bit path: scoring and checking against other programs, a few prompts
        _case("prompt_f32_135m", "smollm2-135m", "prompt", 3, 61, 701, dtype="float32", layers=6),
        # the same path generating for a batch
        _case("decode_f32_360m", "smollm2-360m", "decode", 24, 100, 900, dtype="float32", layers=4),
        # the other designs: prompts and generation
        _case("prompt_sagizen", "sagizen-2048", "prompt", 1, 2048, 2048),
        _case("decode_sagizen", "sagizen-576", "decode", 16, 120, 1500),
        _case("prompt_vosulorn", "vosulorn-576", "prompt", 4, 333, 1700),
        _case("prompt_redenex", "redenex-2048", "prompt", 2, 1000, 2900),
        _case("prompt_radupel", "radupel-576", "prompt", 1, 6000, 6000),
    ]


def draw(rng):
    """One more case: any of the designs and widths, both phases, prompts of 16 to 6,000 tokens, 1 to 64 sequences."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    dtype, layers = "bfloat16", 0
    if rng.random() < 0.5:
        preset = rng.choice(["smollm2-135m", "smollm2-360m", "smollm2-1.7b"])
        layers = rng.randint(2, 4 if preset == "smollm2-1.7b" else 8)
        dtype = "float32" if preset != "smollm2-1.7b" and rng.random() < 0.35 else "bfloat16"
    else:
        preset = rng.choice(["sagizen", "vosulorn", "redenex", "radupel"]) + rng.choice(["-576", "-2048"])
    c = _case("", preset, rng.choice(["prompt", "decode"]), 1, 1, 1, dtype, layers)
    del c["name"]
    if c["phase"] == "decode":
        c["seqs"] = spread(1, 64)
        c["longest"] = spread(64, 2000)
    else:
        c["longest"] = spread(16, 1500 if dtype == "float32" else 6000)
        c["seqs"] = rng.randint(1, max(1, min(12, 8000 // c["longest"] if dtype == "bfloat16" else 2000 // c["longest"])))
    c["shortest"] = c["longest"] if c["seqs"] == 1 else max(1, int(c["longest"] * rng.uniform(0.05, 1.0)))
    return c


def lengths(case):
    """The prompts' lengths: from `shortest` to `longest`, out of order."""
    n, lo, hi = case["seqs"], case["shortest"], case["longest"]
    return [lo + (hi - lo) * ((i * 7) % n if n % 7 else i) // max(1, n - 1) for i in range(n)]


def config_of(case):
    d = copy.deepcopy(PRESETS[case["preset"]])
    picked = DESIGN_LAYERS.get(case["preset"].split("-")[0])
    if picked is None:
        d["num_hidden_layers"] = case["layers"] or d["num_hidden_layers"]
    else:
        d["layers"] = [d["layers"][i] for i in picked]
        d.pop("loop", None)
        for layer in d["layers"]:
            if layer["mlp"]["kind"] == "moe":
                layer["mlp"] = None
    return d


# ----------------------------------------------------------------------------- weights and tokens
def weights_of(case, expected, seed):
    """Weights as a trained model has them where it matters: matrices that keep a vector's size, norms around 1, states that
    remember tens to hundreds of tokens, blends anywhere between a token and the one before it."""
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(shape, mean, std):
        return torch.randn(shape, generator=g, device=DEVICE) * std + mean

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=g, device=DEVICE) * (hi - lo) + lo
    out = {}
    for name, shape in expected.items():
        shape, last = tuple(shape), name.split(".")[-1]
        if last == "A_log":
            t = uniform(shape, 0.0, math.log(8.0))
        elif last == "dt_bias":      # (the step's softplus is then about 0.02 to 0.1)
            t = uniform(shape, -4.0, -2.3)
        elif last == "w0":           # (a decay of exp(-exp(w0)))
            t = uniform(shape, -5.0, -2.0)
        elif last == "lam":
            t = uniform(shape, -5.0, -2.0)
        elif last == "shift" or ".mu." in name:
            t = uniform(shape, 0.0, 1.0)
        elif last in ("lq1", "lk1", "lq2", "lk2", "b", "u", "sink"):
            t = normal(shape, 0.0, 0.1)
        elif last == "conv":
            t = normal(shape, 0.0, 0.5)
        elif ".hc" in name:          # residual streams: read as a mean, mixed by nearly the identity
            streams = shape[0]
            t = normal(shape, 1.0 / streams, 0.05) if last == "in" else normal(shape, 1.0, 0.05) if last == "out" else \
                torch.eye(streams, device=DEVICE) + normal(shape, 0.0, 0.05)
        elif "norm" in last or last == "D" or last in ("input_layernorm", "weight") and len(shape) == 1:
            mean = 0.0 if case["preset"].startswith("redenex") else 1.0      # (that design's norms multiply by 1 + weight)
            t = normal(shape, mean, 0.1)
        else:
            t = normal(shape, 0.0, shape[-1] ** -0.5)
        out[name] = t.to(DTYPES[case["dtype"]])
    return out


def tokens_of(case, seed, vocab):
    g = torch.Generator().manual_seed(int(seed) + 1)
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lengths(case)]
    return prompts, torch.randint(0, vocab, (case["seqs"],), generator=g).tolist()


def wanted(n):
    return sorted(set(range(WANT_EVERY - 1, n, WANT_EVERY)) | {n - 1})


# ----------------------------------------------------------------------------- one pass
def _start_requests(state):
    engine = state["engine"]
    slots = engine.open(len(state["prompts"]))
    for slot, prompt in zip(slots, state["prompts"]):
        engine.step([StepEntry(slot, prompt, [])])
    state["slots"] = slots


def prepare(case, seed):
    config = config_class_for(config_of(case)).from_dict(config_of(case))
    model = DecoderModel(config.plan(), DTYPES[case["dtype"]])
    model.load(weights_of(case, model.expected_weights(), seed), DEVICE)
    prompts, nexts = tokens_of(case, seed, model.plan.vocab_size)
    decode = case["phase"] == "decode"
    most = MAX_POSITIONS if decode else case["longest"]
    most = max(most, WANT_EVERY)
    room = case["seqs"] * most if not decode else min(case["seqs"] * MAX_POSITIONS, 1 << 18)
    engine = Engine(model, max_tokens=(room + 64 * case["seqs"]), max_step_tokens=8192, max_seqs=case["seqs"])
    state = {"engine": engine, "prompts": prompts, "phase": case["phase"]}
    if decode:
        # (as far as every sequence may grow before the requests end and others take their place)
        state["limit"] = min(MAX_POSITIONS, room // case["seqs"]) - 1
        state["next"] = nexts
        _start_requests(state)
    else:
        state["want"] = [wanted(len(p)) for p in prompts]
    return state


def _kept(groups, names):
    """The engine's own tensors of what its sequences keep (a closed sequence's rows stay as they are until others take them)."""
    return [[getattr(g, n) for n in names if getattr(g, n, None) is not None] for g in groups]


def run(state):
    engine = state["engine"]
    cache = engine.cache
    if state["phase"] == "prompt":
        slots = engine.open(len(state["prompts"]))
        logits = engine.step([StepEntry(s, p, w) for s, p, w in zip(slots, state["prompts"], state["want"])])
        engine.close(slots)
        return {"logits": logits, "cache": _kept(cache.kv_groups, ("k", "v", "pooled_k", "pooled_v")), "states": _kept(cache.state_groups, ("state",))}
    if max(engine.length(s) for s in state["slots"]) >= state["limit"]:
        engine.close(state["slots"])
        _start_requests(state)
    return {"logits": engine.decode_launch(state["slots"], state["next"], GREEDY)["logits"], "states": _kept(cache.state_groups, ("state",))}


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Every weight read once, every cached key and value that a token sees read once, the logits written; a matrix
    product's and an attention's two operations per multiply-add."""
    d = config_of(case)
    config = config_class_for(d).from_dict(d)
    model = DecoderModel(config.plan(), DTYPES[case["dtype"]])
    item = 2 if case["dtype"] == "bfloat16" else 4
    lens = lengths(case)
    decode = case["phase"] == "decode"
    shapes = model.expected_weights()
    rows = case["seqs"] if decode else sum(len(wanted(n)) for n in lens)
    tokens = case["seqs"] if decode else sum(lens)
    vocab, width = model.plan.vocab_size, model.plan.hidden_size
    embedding = [n for n in shapes if n.split(".")[0] in ("embed", "model") and tuple(shapes[n]) == (vocab, width)]
    size = sum(math.prod(s) for n, s in shapes.items() if n not in embedding)
    tied = not any(n not in embedding and tuple(s) == (vocab, width) for n, s in shapes.items())
    moved = size + (vocab * width if tied else 0) + tokens * width
    kept = 0      # cache and state bytes
    flops = 2.0 * rows * vocab * width
    layers = d["layers"] if "layers" in d else [{"type": "llama"}] * d["num_hidden_layers"]
    pairs = sum((n + 1) if decode else n * (n + 1) // 2 for n in lens)
    seen = sum(n + 1 if decode else n for n in lens)
    matrices = sum(math.prod(s) for n, s in shapes.items() if len(s) == 2 and tuple(s) != (vocab, width))
    flops += 2.0 * tokens * matrices
    for layer in layers:
        kind, m = layer["type"], layer.get("mixer")
        if kind == "llama":
            h, g, e = d["num_attention_heads"], d["num_key_value_heads"], d["head_dim"]
            kept += seen * 2 * g * e * item
            flops += 4.0 * pairs * h * e
        elif kind == "mamba2":
            kept += case["seqs"] * m["heads"] * m["vdim"] * m["state"] * 8
            flops += 4.0 * tokens * m["heads"] * m["vdim"] * m["state"]
        elif kind == "delta":
            kept += case["seqs"] * m["heads"] * m["dim"] * m["vdim"] * 8
            flops += 6.0 * tokens * m["heads"] * m["dim"] * m["vdim"]
        elif kind == "rglru":
            kept += case["seqs"] * m["width"] * 8
            flops += 4.0 * tokens * m["width"] * m["width"] / m["blocks"]
        elif kind == "latent_attention":
            kept += seen * (m["kv_rank"] + m["rot_dim"]) * item
            flops += 2.0 * pairs * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        else:
            left = m.get("left", m)
            size_of = (left.get("mask") or {}).get("size")
            pool = (left.get("mask") or {}).get("pool")
            maps = 2 if "diff" in left else 1
            if size_of and pool:         # a window, and a pooled row per block behind it
                see = [[min(i + 1, size_of) + max(0, i + 1 - size_of) // pool for i in ([n] if decode else range(n))] for n in lens]
            elif size_of:                # chunks
                see = [[i % size_of + 1 for i in ([n] if decode else range(n))] for n in lens]
            else:
                see = [[n + 1] if decode else [n * (n + 1) // 2] for n in lens]
            p = sum(map(sum, see))
            kept += (p if decode else seen) * left["kv_heads"] * (maps * left["dim"] + left["vdim"]) * item
            flops += 2.0 * p * left["heads"] * maps * (left["dim"] + left["vdim"])
            if "right" in m:
                r = m["right"]
                kept += case["seqs"] * r["heads"] * r["dim"] * r["dim"] * 8
                flops += 4.0 * tokens * r["heads"] * r["dim"] * r["dim"]
    return {"bytes": float(moved * item + kept + rows * vocab * 4), "flops": float(flops)}


def tolerance(case):
    """About four times what a correct run is off the same in 64 bits (measured: 1e-6 in float32; in bfloat16 0.007 to 0.01
    for the Llama decoder and the Sagizen layers, 0.003 to 0.005 for the other designs' layers)."""
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 2e-4}
    return {"rel": 0.03, "max": 0.3} if case["preset"].startswith(("smollm2", "sagizen")) else {"rel": 0.02, "max": 0.2}


# ----------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w=None, eps=1e-5, plus=0.0):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * (w + plus)


def _silu(z):
    return z * torch.sigmoid(z)


def _shift(h, mu):
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    return h + (before - h) * mu


def _conv(u, taps, bias=None):
    n, k = u.shape[0], taps.shape[1]
    padded = torch.cat([u.new_zeros(k - 1, u.shape[1]), u])
    y = sum(padded[j:j + n] * taps[:, j] for j in range(k))
    return y if bias is None else y + bias


def _rotate(x, dims, base, interleaved=False, scaling=None):
    """x [n, heads, d]: the first `dims` dimensions turned by position * frequency."""
    if not dims:
        return x
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    if scaling and "low" in scaling:       # long wavelengths stretched, short ones kept, a blend between them
        wave = 2.0 * math.pi / f
        s = (scaling["original"] / wave - scaling["low"]) / (scaling["high"] - scaling["low"])
        f = torch.where(wave < scaling["original"] / scaling["high"], f,
                        torch.where(wave > scaling["original"] / scaling["low"], f / scaling["factor"],
                                    (1.0 - s) * f / scaling["factor"] + s * f))
    elif scaling:
        f = f / scaling["factor"]
    ang = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = ang.cos(), ang.sin()
    if interleaved:
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        turned = torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    else:
        a, b = x[..., :half], x[..., half:dims]
        turned = torch.cat([a * c - b * s, b * c + a * s], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, scale, rows, sees=None, sink=None, more=None):
    """q [r, H, d] of the positions `rows`, k [n, G, d], v [n, G, e]; `sees(i, j)`: beside j <= i; `more`: further keys and
    values and whether a row sees them."""
    H, G, at = q.shape[1], k.shape[1], torch.arange(k.shape[0], device=q.device)
    out = q.new_zeros(q.shape[0], H, v.shape[2])
    for a in range(0, q.shape[0], 512):
        i = rows[a:a + 512, None]
        mask = at[None] <= i
        if sees is not None:
            mask = mask & sees(i, at[None])
        for h in range(H):
            g = h // (H // G)
            s = (q[a:a + 512, h] @ k[:, g].T * scale).masked_fill(~mask, -math.inf)
            vals = v[:, g]
            if more is not None and more[0].shape[0]:
                s = torch.cat([s, (q[a:a + 512, h] @ more[0][:, g].T * scale).masked_fill(~more[2](i), -math.inf)], 1)
                vals = torch.cat([vals, more[1][:, g]])
            if sink is not None:
                s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
                vals = torch.cat([vals, torch.zeros_like(vals[:1])])
            out[a:a + 512, h] = torch.softmax(s, -1) @ vals
    return out


def _heads(h, w, b, heads):
    y = h @ w.T
    return (y if b is None else y + b).view(h.shape[0], heads, -1)


def _llama_layer(x, W, p, d):
    H, G, n = d["num_attention_heads"], d["num_key_value_heads"], x.shape[0]
    h = _norm(x, W[p + "input_layernorm.weight"], d["rms_norm_eps"])
    q, k, v = (_heads(h, W[f"{p}self_attn.{s}_proj.weight"], None, m) for s, m in (("q", H), ("k", G), ("v", G)))
    q, k = _rotate(q, d["head_dim"], d["rope_theta"]), _rotate(k, d["head_dim"], d["rope_theta"])
    a = _attend(q, k, v, d["head_dim"] ** -0.5, torch.arange(n, device=x.device))
    x = x + a.reshape(n, -1) @ W[p + "self_attn.o_proj.weight"].T
    h = _norm(x, W[p + "post_attention_layernorm.weight"], d["rms_norm_eps"])
    g, u = h @ W[p + "mlp.gate_proj.weight"].T, h @ W[p + "mlp.up_proj.weight"].T
    return x + (_silu(g) * u) @ W[p + "mlp.down_proj.weight"].T


def _mamba2(h, W, p, m, eps):
    n, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, xbc, dt = (h @ W[p + "in"].T).split([inner, inner + 2 * G * N, H], 1)
    xbc = _silu(_conv(xbc, W[p + "conv"], W[p + "conv.b"]))
    x, B, C = xbc.split([inner, G * N, G * N], 1)
    x = x.reshape(n, H, P)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = torch.nn.functional.softplus(dt + W[p + "dt_bias"])
    keep = torch.exp(-torch.exp(W[p + "A_log"]) * dt)
    S, y = x.new_zeros(H, N, P), torch.empty_like(x)
    B = B * dt[:, :, None]
    for t in range(n):
        S = torch.baddbmm(S * keep[t, :, None, None], B[t, :, :, None], x[t, :, None, :])
        y[t] = torch.bmm(C[t, :, None, :], S)[:, 0]
    y = (y + W[p + "D"][:, None] * x).reshape(n, inner) * _silu(z)
    ng = m["norm_groups"]
    return _norm(y.view(n, ng, -1), eps=eps).reshape(n, inner) * W[p + "norm"] @ W[p + "o"].T


def _pooled_attention(h, W, p, m, eps):
    n, H, G = h.shape[0], m["heads"], m["kv_heads"]
    q, k, v = (_heads(h, W[p + s], W[p + s + ".b"], c) for s, c in (("q", H), ("k", G), ("v", G)))
    rot = m["rot"]
    q, k = (_norm(_rotate(t, rot["dims"], rot["base"], scaling=rot.get("scaling")), eps=eps) for t in (q, k))
    window, pool = m["mask"]["size"], m["mask"]["pool"]
    nb = n // pool
    pk, pv = (t[:nb * pool].view(nb, pool, G, -1).mean(1) for t in (k, v))
    ends = torch.arange(nb, device=h.device)[None] * pool + pool - 1
    o = _attend(q, k, v, m["scale"], torch.arange(n, device=h.device), lambda i, j: i - j < window,
                more=(pk, pv, lambda i: ends <= i - window))
    return o.reshape(n, -1) @ W[p + "o"].T


def _time_mix(h, W, p, m, eps):
    n, H, K = h.shape[0], m["heads"], m["dim"]
    b = {s: _shift(h, W[p + "mu." + s]) for s in "rkvgw"}
    r, k, v = ((b[s] @ W[p + s].T).view(n, H, K) for s in "rkv")
    gate = _silu(b["g"] @ W[p + "g"].T)
    w = torch.exp(-torch.exp(torch.tanh(b["w"] @ W[p + "w1"].T) @ W[p + "w2"].T + W[p + "w0"])).view(n, H, K)
    S, o = h.new_zeros(H, K, K), torch.empty_like(r)
    for t in range(n):
        o[t] = torch.bmm(r[t, :, None, :], S)[:, 0]
        S = torch.baddbmm(S * w[t, :, :, None], k[t, :, :, None], v[t, :, None, :])
    o = o + (r * W[p + "u"] * k).sum(-1, keepdim=True) * v
    return (_norm(o, eps=eps).reshape(n, H * K) * W[p + "norm"] * gate) @ W[p + "o"].T


def _sagizen_layer(x, W, p, layer, eps):
    h, m = _shift(x, W[p + "shift"]), layer["mixer"]
    if layer["type"] == "mamba2":
        y = _mamba2(h, W, p + "mix.", m, eps)
    else:
        y = m["left_scale"] * _pooled_attention(h, W, p + "mix.left.", m["left"], eps) + \
            m["right_scale"] * _time_mix(h, W, p + "mix.right.", m["right"], eps)
    x = x + _norm(y, W[p + "norm1"], eps)
    f = (_silu(x @ W[p + "mlp.gate"].T) * (x @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T
    return x + _norm(f, W[p + "norm2"], eps)


def _delta(h, W, p, m, eps):
    n, H, G = h.shape[0], m["heads"], m["kv_heads"]
    q, k, v = (_silu(_conv(h @ W[p + s].T, W[p + s + ".conv"])).view(n, c, -1) for s, c in (("q", G), ("k", G), ("v", H)))
    q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(H // G, 1) for t in (q * m["dim"] ** -0.5, k))
    beta = torch.sigmoid(h @ W[p + "b"].T)
    g = torch.exp(-torch.exp(W[p + "A_log"]) * torch.nn.functional.softplus(h @ W[p + "a"].T + W[p + "dt_bias"]))
    S, o = h.new_zeros(H, m["dim"], m["vdim"]), torch.empty_like(v)
    for t in range(n):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None, :])
        o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    o = (_norm(o, eps=eps) * W[p + "norm"]).reshape(n, -1)
    return (o * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T


def _chunked_attention(h, W, p, m, eps):
    n, H, G = h.shape[0], m["heads"], m["kv_heads"]
    q, k, v = (_heads(h, W[p + s], W[p + s + ".b"], c) for s, c in (("q", H), ("k", G), ("v", G)))
    rot, size = m["rot"], m["mask"]["size"]
    q, k = (_rotate(t, rot["dims"], rot["base"], True, rot.get("scaling")) for t in (q, k))
    o = _attend(q, k, v, m["scale"], torch.arange(n, device=h.device), lambda i, j: i // size == j // size, sink=W[p + "sink"])
    return o.reshape(n, -1) @ W[p + "o"].T + W[p + "o.b"]


def _latent_attention(h, W, p, m, eps):
    n, H, r, rd = h.shape[0], m["heads"], m["kv_rank"], m["rot_dim"]
    ckr, base = h @ W[p + "dkv"].T, m["rot"]["base"]
    c = _norm(ckr[:, :r], W[p + "dkv.norm"], eps)
    kr = _rotate(ckr[:, None, r:], rd, base)
    q = (h @ W[p + "q"].T).view(n, H, -1)
    q = torch.cat([q[..., :-rd], _rotate(q[..., -rd:], rd, base)], -1)
    k = torch.cat([(c @ W[p + "uk"].T).view(n, H, -1), kr.expand(n, H, rd)], -1)
    o = _attend(q, k, (c @ W[p + "uv"].T).view(n, H, -1), m["scale"], torch.arange(n, device=h.device))
    return o.reshape(n, -1) @ W[p + "o"].T


def _vosulorn_layer(x, W, p, layer, eps):
    mixer = {"delta": _delta, "attention": _chunked_attention, "latent_attention": _latent_attention}[layer["type"]]
    return x + mixer(_norm(x, W[p + "norm1"], eps), W, p + "mix.", layer["mixer"], eps)


def _rglru(h, W, p, m, eps):
    n, blocks = h.shape[0], m["blocks"]
    y = torch.nn.functional.gelu(h @ W[p + "y"].T + W[p + "y.b"], approximate="tanh")
    u = _conv(h @ W[p + "x"].T + W[p + "x.b"], W[p + "conv"], W[p + "conv.b"])
    r, i = (torch.sigmoid(torch.einsum("bok,nbk->nbo", W[p + s], u.view(n, blocks, -1)) + W[p + s + ".b"]).reshape(n, -1) for s in ("ra", "ri"))
    a = torch.exp(-8.0 * r * torch.nn.functional.softplus(W[p + "lam"]))
    b = torch.sqrt(1.0 - a * a) * i * u
    S, out = torch.zeros_like(u[0]), torch.empty_like(u)
    for t in range(n):
        S = torch.addcmul(b[t], a[t], S)
        out[t] = S
    return (out * y) @ W[p + "o"].T


def _two_maps(h, W, p, m, eps):
    n, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (_conv(h @ W[p + s].T + W[p + s + ".b"], W[p + s + ".conv"]) for s in "qkv")
    q = _norm(q.view(n, H * 2, d), W[p + "q.norm"], eps)
    k = _norm(k.view(n, G * 2, d), W[p + "k.norm"], eps)
    rot, size = m["rot"], m["mask"]["size"]
    q, k = (_rotate(t, rot["dims"], rot["base"]).view(n, -1, 2, d) for t in (q, k))
    a1, a2 = (_attend(q[:, :, j], k[:, :, j], v.view(n, G, -1), m["scale"], torch.arange(n, device=h.device),
                      lambda i, j: i // size == j // size) for j in range(2))
    lam = torch.exp((W[p + "lq1"] * W[p + "lk1"]).sum()) - torch.exp((W[p + "lq2"] * W[p + "lk2"]).sum()) + m["diff"]
    o = _norm(a1 - lam * a2, eps=eps) * (1.0 - m["diff"])
    return o.reshape(n, -1) @ W[p + "o"].T


def _redenex_layer(xs, W, p, layer, eps):
    """xs [streams, n, width]"""
    def sublayer(xs, pre, fn):
        y = fn(torch.einsum("s,snd->nd", W[pre + "in"], xs))
        return torch.einsum("st,snd->tnd", W[pre + "mix"], xs) + W[pre + "out"][:, None, None] * y
    mixer, limit = {"rglru": _rglru, "attention": _two_maps}[layer["type"]], layer["mlp"]["limit"]

    def ff(u):
        h = _norm(u, W[p + "norm2"], eps, 1.0)
        g, up = (h @ W[p + "mlp.gate"].T).clamp(max=limit), (h @ W[p + "mlp.up"].T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (up + 1.0)) @ W[p + "mlp.down"].T
    xs = sublayer(xs, p + "hc1.", lambda u: mixer(_norm(u, W[p + "norm1"], eps, 1.0), W, p + "mix.", layer["mixer"], eps))
    return sublayer(xs, p + "hc2.", ff)


def _radupel_layer(x, W, p, layer, eps):
    h, h2, m = _norm(x, W[p + "norm1"], eps), _norm(x, W[p + "norm2"], eps), layer["mixer"]
    left, right, n, a = m["left"], m["right"], x.shape[0], p + "mix.left."
    q, k, v = (_conv(h @ W[a + s].T, W[a + s + ".conv"]) for s in "qkv")
    q, k, v = q.view(n, left["heads"], -1), k.view(n, left["kv_heads"], -1), v.view(n, left["kv_heads"], -1)
    q, k = (_rotate(t, left["rot"]["dims"], left["rot"]["base"]) for t in (q, k))
    o = _attend(q, k, v, left["scale"], torch.arange(n, device=x.device)) * torch.sigmoid(h @ W[a + "g"].T)[:, :, None]
    y = m["left_scale"] * (o.reshape(n, -1) @ W[a + "o"].T)
    b = p + "mix.right."
    q, k, v = (_silu(h @ W[b + s].T).view(n, right["heads"], -1) for s in "qkv")
    S, o = x.new_zeros(right["heads"], right["dim"], right["vdim"]), torch.empty_like(v)
    decay = torch.tensor(right["decay"], dtype=torch.float64, device=x.device)[:, None, None]
    for t in range(n):
        S = torch.baddbmm(S * decay, k[t, :, :, None], v[t, :, None, :])
        o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    o = _norm(o.reshape(n, -1), W[b + "norm"], eps) * torch.sigmoid(h @ W[b + "g"].T)
    y = y + m["right_scale"] * (o @ W[b + "o"].T)
    g, u = h2 @ W[p + "mlp.gate"].T + W[p + "mlp.gate.b"], h2 @ W[p + "mlp.up"].T + W[p + "mlp.up.b"]
    return x + y + (_silu(g) * u) @ W[p + "mlp.down"].T + W[p + "mlp.down.b"]


def _logits(d, W, ids, rows):
    design = d.get("architecture", "llama").lower()
    ids = torch.tensor(ids, device=DEVICE)
    if design == "llama":
        x, eps, head = W["model.embed_tokens.weight"][ids], d["rms_norm_eps"], W["model.embed_tokens.weight"]
        for i in range(d["num_hidden_layers"]):
            x = _llama_layer(x, W, f"model.layers.{i}.", d)
        return _norm(x[rows], W["model.norm.weight"], eps) @ head.T
    eps, x = d["norm"]["eps"], W["embed"][ids] * d.get("embedding", {}).get("scale", 1.0)
    layer = {"sagizen": _sagizen_layer, "vosulorn": _vosulorn_layer, "redenex": _redenex_layer, "radupel": _radupel_layer}[design]
    if design == "redenex":
        x = x.expand(d["streams"], *x.shape)
    for i, spec in enumerate(d["layers"]):
        x = layer(x, W, f"l{i}.", spec, eps)
    if design == "redenex":
        x = x.sum(0)
    y = _norm(x[rows], W["final.norm"], eps, 1.0 if design == "redenex" else 0.0) @ W.get("head", W["embed"]).T
    cap = d.get("logit_softcap")
    return cap * torch.tanh(y / cap) if cap else y


def exact(case, seed):
    """Every sequence's logits from its start in float64, without a cache, from the weights in the dtype that the model holds."""
    d = config_of(case)
    plan = config_class_for(d).from_dict(d).plan()
    expected = DecoderModel(plan, DTYPES[case["dtype"]]).expected_weights()
    W = {k: t.double() for k, t in weights_of(case, expected, seed).items()}
    prompts, nexts = tokens_of(case, seed, plan.vocab_size)
    out = []
    for p, t in zip(prompts, nexts):
        ids = p + [t] if case["phase"] == "decode" else p
        rows = torch.tensor([len(p)] if case["phase"] == "decode" else wanted(len(p)), device=DEVICE)
        out.append(_logits(d, W, ids, rows))
    return {"logits": torch.cat(out)}
