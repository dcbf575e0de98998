"""The steps that programs run through `Engine.step`, as cases to be timed and compared.

A case is what an inference program has the engine do once: one decode step of some requests, the prompts of new
requests (whole or in portions), or prompts in portions beside requests that decode (continuous batching). A pass
gives the engine host token ids and gets float logits back; prompts are ended after the pass, requests that decode
go on, so that the next pass is their next token.

The models are the Llama 1B shape (16 layers; the benchmark's default) and the four-layer models that the benchmark
times for five of the other designs, with random weights. Feed-forwards are dense here: a router's choice flips with
the last bit of its input, so that logits of a model with routed experts, summed in another order, say nothing about
precision. bfloat16 throughout, as these models are served; the 32-bit run is there to be compared with.
"""
import math

import torch

from rllm_b200.config import config_from_dict
from rllm_b200.engine import Entry, random_engine
from rllm_b200.weights.loader import expected_tensors

DEVICE = "cuda:0"
PAGE = 16
ROOM = 4096          # tokens that a decoding request may grow by before it is begun again
FILL = 2048          # tokens of a context that one step brings in

LLAMA = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": 2048, "num_hidden_layers": 16,
    "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64, "intermediate_size": 8192,
    "vocab_size": 128256, "max_position_embeddings": 131072, "rope_theta": 500000.0, "rms_norm_eps": 1e-5,
    "tie_word_embeddings": True,
    "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                     "original_max_position_embeddings": 8192}}


def config(model, width):
    """The raw configuration. The four-layer models have heads of 128 (Livovik of 64 at width 2,048)."""
    W, H = width, width // 128
    yarn = {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    if model == "llama":
        return LLAMA
    if model == "livovik":
        D, heads = (64, 32) if W == 2048 else (128, 32)
        mixer = {"heads": heads, "kv_heads": 8, "dim": D, "vdim": D, "scale": D ** -0.5, "mask": {"size": 8192},
                 "rot": {"base": 500000.0, "dims": D // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        layer = {"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": 12288 if W == 2048 else 21504}}
        return {"architecture": "Livovik", "vocab": 32000, "width": W, "norm": {"eps": 1e-6}, "postln_alpha": 2.0,
                "layers": [layer] * 4}
    att = {"heads": H, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    if model == "bazulorn":
        ff = {"kind": "dense", "ff": 8 * W // 3 // 64 * 64}
        par = {"type": "parallel", "mlp": ff, "mixer": {
            "left": dict(att, mask={"size": 4096}),
            "right": {"heads": W // 64, "vdim": 64, "state": 128, "groups": 4, "norm_groups": 4, "conv": 4}}}
        rec = {"type": "channel_delta", "mlp": ff,
               "mixer": {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 16, "gate_rank": 64}}
        return {"architecture": "Bazulorn", "vocab": 32000, "width": W, "norm": {"eps": 1e-6}, "layers": [par, rec, rec, par]}
    ff = {"kind": "dense", "ff": 4 * W}
    if model == "purozen":
        win = {"type": "attention", "mlp": ff, "mixer": dict(
            att, mask={"size": 1024, "keep_first": 64}, rot={"base": 1000000.0, "dims": 64, "scaling": {"factor": 4.0}}, v_mix=True)}
        par = {"type": "parallel", "mlp": ff, "mixer": {"left": att, "left_scale": 0.5, "right": {"width": W}, "right_scale": 0.5}}
        lat = {"type": "latent_attention", "mlp": ff,
               "mixer": {"heads": H, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5}}
        return {"architecture": "Purozen", "vocab": 32000, "width": W, "norm": {"eps": 1e-6}, "layers": [par, win, lat, win]}
    if model == "danonex":
        soft = {"type": "attention", "mlp": ff, "mixer": dict(att, softcap=30.0, rot={"base": 1000000.0, "dims": 64, "scaling": yarn})}
        rec = {"type": "delta", "mlp": ff, "mixer": {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4}}
        return {"architecture": "Danonex", "vocab": 32000, "width": W, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
                "logit_scale": 2.0, "layers": [soft, rec, rec, soft]}
    if model == "zufotar":
        lat = {"type": "latent_attention", "mlp": ff, "mixer": {
            "heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 1536, "kv_rank": 512, "scale": 192 ** -0.5,
            "rot": {"base": 10000.0, "dims": 64, "scaling": dict(yarn, factor=4.0)}}}
        rec = {"type": "wkv", "mlp": ff, "mixer": {"heads": H, "dim": 128, "decay_rank": 64}}
        return {"architecture": "Zufotar", "vocab": 32000, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
                "logit_softcap": 30.0, "layers": [lat, rec, rec, lat]}
    raise ValueError(model)


# ------------------------------------------------------------------ the cases

def _case(name, model, width=2048, decoding=0, context=0, prompts=0, tokens=0, portion=0):
    """`decoding` requests whose contexts reach from an eighth of `context` up to it; `prompts` new ones whose lengths
    reach from an eighth of `tokens` up to it (one alone has it), brought in portions of `portion` tokens (0: whole)."""
    return {"name": name, "model": model, "width": width, "decoding": decoding, "context": context, "prompts": prompts,
            "tokens": tokens, "portion": portion}


def listed():
    return [
        # one user's chat: a token at a time, the latency of a step
        _case("llama decode 1", "llama", decoding=1, context=700),
        # a small batch at long context: the benchmark's headline point
        _case("llama decode 8", "llama", decoding=8, context=4090),
        # a full server: contexts of all lengths
        _case("llama decode 64", "llama", decoding=64, context=2040),
        # a prompt in one step: the benchmark's prefill point
        _case("llama prompt", "llama", prompts=1, tokens=2048),
        # a long document in the scheduler's portions of 2,048: later portions read the cache of the earlier ones
        _case("llama long prompt", "llama", prompts=1, tokens=6001, portion=2048),
        # continuous batching: requests decode while two prompts come in by portions of 512
        _case("llama mixed", "llama", decoding=24, context=1500, prompts=2, tokens=1100, portion=512),
        # prompts of the other designs, each with its own mixers: whole, ragged and odd, at both of the benchmark's widths
        _case("livovik prompt", "livovik", prompts=1, tokens=2048),
        _case("bazulorn prompt", "bazulorn", prompts=1, tokens=2048),
        _case("purozen prompts", "purozen", prompts=3, tokens=1333),
        _case("danonex prompt", "danonex", width=4096, prompts=1, tokens=2047),
        _case("zufotar prompt", "zufotar", prompts=1, tokens=2048),
        # decoding over recurrent states and attention caches together
        _case("bazulorn decode 8", "bazulorn", decoding=8, context=1100),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["llama", "llama", "llama", "livovik", "bazulorn", "purozen", "danonex", "zufotar"])
    width = 2048 if model == "llama" or rng.random() < 0.6 else 4096
    kind = rng.choice(["decode", "prompt", "prompt", "mixed"])
    case = _case("", model, width)
    del case["name"]
    if kind in ("decode", "mixed"):
        case["decoding"] = log(1, 64) if kind == "decode" else log(2, 24)
        case["context"] = log(64, 4096 if case["decoding"] <= 8 else 2040)
    if kind in ("prompt", "mixed"):
        case["prompts"] = rng.choice([1, 1, 2, 3, 4])
        case["tokens"] = log(48, (4096 if model == "llama" and case["prompts"] == 1 else 2048) // (1 if case["prompts"] < 3 else 2))
        case["portion"] = rng.choice([256, 512]) if kind == "mixed" else rng.choice([0, 0, 1024])
    return case


def _lengths(n, longest):
    """n lengths from `longest` down to an eighth of it."""
    return [max(1, longest - longest * 7 * i // (8 * n)) for i in range(n)]


def _portions(case):
    """Per step of a pass: [(prompt, begin, end)]."""
    steps = []
    for p, n in enumerate(_lengths(case["prompts"], case["tokens"])):
        size = case["portion"] or n
        for k, at in enumerate(range(0, n, size)):
            while len(steps) <= k:
                steps.append([])
            steps[k].append((p, at, min(n, at + size)))
    return steps or [[]]


def _inputs(case, seed):
    """Token ids: the decoding requests' contexts, what they decode in turn, the prompts."""
    cfg = config(case["model"], case["width"])
    g = torch.Generator().manual_seed(seed)
    ids = lambda n: torch.randint(0, cfg.get("vocab", cfg.get("vocab_size")), (n,), generator=g).tolist()
    return ([ids(n) for n in _lengths(case["decoding"], case["context"])], [ids(64) for _ in range(case["decoding"])],
            [ids(n) for n in _lengths(case["prompts"], case["tokens"])])


def _fill(state):
    eng = state["engine"]
    for i, ids in enumerate(state["contexts"]):
        for at in range(0, len(ids), FILL):
            eng.step([Entry(("d", i), ids[at: at + FILL], [])])
    state["grown"] = 0


def prepare(case, seed):
    contexts, decoded, prompts = _inputs(case, seed)
    pages = sum((len(c) + ROOM) // PAGE + 2 for c in contexts) + sum(len(p) // PAGE + 2 for p in prompts)
    eng = random_engine(config(case["model"], case["width"]), seed, dtype="bfloat16", device=DEVICE, page_size=PAGE,
                        num_pages=pages + 16, max_requests=case["decoding"] + case["prompts"] + 1)
    state = {"engine": eng, "contexts": contexts, "decoded": decoded, "prompts": prompts, "steps": _portions(case)}
    _fill(state)
    return state


def run(state):
    eng, steps = state["engine"], state["steps"]
    if state["contexts"] and state["grown"] + len(steps) > ROOM:      # these requests are over; others like them begin
        eng.end([("d", i) for i in range(len(state["contexts"]))])
        _fill(state)
    out = []
    for step in steps:
        entries = [Entry(("d", i), [ids[state["grown"] % len(ids)]], [0]) for i, ids in enumerate(state["decoded"])]
        for p, a, b in step:
            ids = state["prompts"][p]
            entries.append(Entry(("p", p), ids[a:b], [b - a - 1] if b == len(ids) else []))
        logits = eng.step(entries)
        if logits is not None:
            out.append(logits)
        state["grown"] += 1
    if state["prompts"]:
        eng.end([("p", p) for p in range(len(state["prompts"]))])
    return out


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(case):
    """(elements of the matrices that every token meets, elements of the output matrix, numbers of a cached position that a
    token reads, multiplications a token and cached position, numbers of a request's recurrent states, width, vocabulary)."""
    cfg = config(case["model"], case["width"])
    arch, typed = config_from_dict(cfg)
    body = sum(math.prod(s.shape) for name, s, p, _ in expected_tensors(arch.build(typed))
               if p.role == "matrix" and "embed" not in name and name != "head")
    if case["model"] == "llama":
        L, q, kv = cfg["num_hidden_layers"], cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
        return body, cfg["hidden_size"] * cfg["vocab_size"], L * 2 * kv, L * 2 * q, 0, cfg["hidden_size"], cfg["vocab_size"]
    keys = pairs = states = 0
    for layer in cfg["layers"]:
        m = layer["mixer"]
        m, other = (m["left"], m["right"]) if layer["type"] == "parallel" else (m, None)
        if layer["type"] == "latent_attention":
            keys += m["kv_rank"] + m.get("rot_dim", 0)
            pairs += m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])
        elif layer["type"] in ("attention", "parallel"):
            keys += m["kv_heads"] * (m["dim"] + m["vdim"])
            pairs += m["heads"] * (m["dim"] + m["vdim"])
        else:
            states += m["heads"] * m["dim"] * m.get("vdim", m["dim"])
        if other is not None:
            states += other.get("width", 0) + other.get("heads", 0) * other.get("vdim", 0) * other.get("state", 0)
    return body, cfg["width"] * cfg["vocab"], keys, pairs, states, cfg["width"], cfg["vocab"]


def work(case):
    body, head, keys, pairs, states, width, vocab = _sizes(case)
    prompts, contexts = _lengths(case["prompts"], case["tokens"]), _lengths(case["decoding"], case["context"])
    total = flops = 0
    for step in _portions(case):
        ends = sum(b == prompts[p] for p, _, b in step)
        tokens, rows = case["decoding"] + sum(b - a for _, a, b in step), case["decoding"] + ends
        seen = sum(contexts) + sum(a for _, a, _ in step)               # cached positions read
        scored = sum(contexts) + sum((b - a) * (a + b + 1) // 2 for _, a, b in step)
        total += 2 * body + (2 * head if rows else 0) + 2 * keys * (seen + tokens) + 2 * 4 * states * (case["decoding"] + len(step))
        total += 2 * width * tokens + 4 * vocab * rows
        flops += 2 * body * tokens + 2 * head * rows + 2 * pairs * scored + 6 * states * tokens
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """bfloat16 rounds weights, activations and caches to 8 bits and a model's layers add up what that leaves. Logits are
    a sum over the whole width, so one value's difference is of the size of the norm's. Measured against 64 bits: 0.004 to
    0.007 for four layers of Livovik, Purozen and Zufotar, 0.007 to 0.011 for Bazulorn and Danonex, 0.015 to 0.019 for the
    sixteen Llama layers."""
    return {"rel": 0.02 if case["model"] in ("livovik", "purozen", "zufotar") else 0.03, "max": 0.2}


# ------------------------------------------------------------------ the same in 64 bits

F64 = torch.float64


def _weights(cfg, seed):
    """name -> the random-weights mode's tensor as bfloat16 stores it, in 64 bits: drawn in the order the model lists them."""
    arch, typed = config_from_dict(cfg)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    w = {}
    for name, s, _, _ in expected_tensors(arch.build(typed)):
        if s.init == "normal":
            t = torch.randn(s.shape, generator=g, dtype=torch.float32, device=DEVICE) * 0.02
        else:
            t = torch.full(s.shape, float(s.init == "norm"), device=DEVICE)
        w[name] = t.bfloat16().to(F64)
    return w


def _rms(x, w=None, eps=1e-6):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu_tanh(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _gelu_erf(z):
    return 0.5 * z * (1 + torch.erf(z / math.sqrt(2.0)))


def _angles(T, base, dims, rule=None):
    """cos and sin [T, 1, dims/2] of a rotation; `rule` changes its frequencies and gives a factor."""
    f = [float(base) ** (-2.0 * i / dims) for i in range(dims // 2)]
    mag = 1.0
    if rule and "fast" in rule:                                     # yarn
        at = lambda turns: dims * math.log(rule["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(at(rule["fast"])), 0), min(math.ceil(at(rule["slow"])), dims - 1)
        for i in range(dims // 2):
            r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            f[i] = f[i] / rule["factor"] * r + f[i] * (1 - r)
        mag = 0.1 * math.log(rule["factor"]) + 1.0
    elif rule and "low" in rule:                                    # bands of wavelengths
        for i in range(dims // 2):
            wave = 2 * math.pi / f[i]
            if wave > rule["original"] / rule["low"]:
                f[i] /= rule["factor"]
            elif wave >= rule["original"] / rule["high"]:
                s = (rule["original"] / wave - rule["low"]) / (rule["high"] - rule["low"])
                f[i] = (1 - s) * f[i] / rule["factor"] + s * f[i]
    elif rule:
        f = [x / rule["factor"] for x in f]
    a = torch.arange(T, dtype=F64, device=DEVICE)[:, None] * torch.tensor(f, dtype=F64, device=DEVICE)
    return torch.cos(a)[:, None] * mag, torch.sin(a)[:, None] * mag


def _turn_halves(x, cs):
    c, s = cs
    n = c.shape[-1]
    u, v = x[..., :n], x[..., n: 2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _turn_pairs(x, cs):
    c, s = cs
    n = c.shape[-1]
    u, v = x[..., 0: 2 * n: 2], x[..., 1: 2 * n: 2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., 2 * n:]], -1)


def _seen(T, window=None, first=0, block=None):
    i = torch.arange(T, device=DEVICE)
    q, k = i[:, None], i[None, :]
    ok = k <= q
    if window is not None:
        ok &= (q - k < window) | (k < first)
    if block is not None:
        ok &= q // block == k // block
    return ok


def _softmax_weights(s, ok, sink=None):
    """Over the last dimension of s [heads, T, T]; `sink` [heads]: exp(sink) in the denominator too."""
    s = s.masked_fill_(~ok, -math.inf)
    if sink is None:
        return torch.softmax(s, -1)
    m = torch.maximum(s.amax(-1, keepdim=True), sink[:, None, None])
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + torch.exp(sink[:, None, None] - m))


def _attend(q, k, v, weights):
    """q [T, H, d], k, v [T, G, d]: head by head of G; `weights(scores [n, T, T], heads)` are what the values are summed by."""
    T, H, _ = q.shape
    G = k.shape[1]
    n = H // G
    out = []
    for g in range(G):
        a = weights(torch.einsum("ihd,jd->hij", q[:, g * n: (g + 1) * n], k[:, g]), slice(g * n, (g + 1) * n))
        out.append(torch.einsum("hij,jd->ihd", a, v[:, g]))
    return torch.cat(out, 1).reshape(T, -1)


def _conv(x, w, b=None):
    """A causal convolution per channel; w [C, taps], its last column meets the current token."""
    T, taps = x.shape[0], w.shape[1]
    padded = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=F64, device=DEVICE), x])
    y = sum(w[:, j] * padded[j: j + T] for j in range(taps))
    return y if b is None else y + b


def _delta(q, k, v, decay, beta):
    """q, k, decay [T, H, d] (decay of 1 or d channels), v [T, H, dv], beta [T, H]."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F64, device=DEVICE)
    out = torch.empty_like(v)
    for t in range(k.shape[0]):
        S *= decay[t][:, :, None]
        u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S += k[t][:, :, None] * u[:, None]
        out[t] = (q[t][:, None] @ S)[:, 0]
    return out


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _delta_mixer(n, w, p, m, eps, per_channel):
    T, H, G, d, dv = n.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_silu(_conv(n @ w[p + c].T, w[p + c + ".conv"])).view(T, -1, d) for c in "qkv")
    q, k = _unit(q) * d ** -0.5, _unit(k)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    z = (n @ w[p + "a1"].T) @ w[p + "a2"].T if per_channel else n @ w[p + "a"].T
    step = torch.nn.functional.softplus(z + w[p + "dt_bias"], threshold=60).view(T, H, -1)
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * step)
    o = _rms(_delta(q, k, v.view(T, H, dv), decay, torch.sigmoid(n @ w[p + "b"].T)), w[p + "norm"], eps).reshape(T, -1)
    gate = torch.sigmoid((n @ w[p + "g1"].T) @ w[p + "g2"].T) if per_channel else _silu(n @ w[p + "g"].T)
    return (o * gate) @ w[p + "o"].T


def _llama(cfg, w, ids):
    L, H, G, D, eps = (cfg[k] for k in ("num_hidden_layers", "num_attention_heads", "num_key_value_heads", "head_dim", "rms_norm_eps"))
    sc = cfg["rope_scaling"]
    cs = _angles(len(ids), cfg["rope_theta"], D, {"factor": sc["factor"], "low": sc["low_freq_factor"], "high": sc["high_freq_factor"],
                                                  "original": sc["original_max_position_embeddings"]})
    x, T = w["model.embed_tokens.weight"][ids], len(ids)
    ok = _seen(T)
    for i in range(L):
        p = "model.layers.%d." % i
        n = _rms(x, w[p + "input_layernorm.weight"], eps)
        q, k, v = ((n @ w[p + "self_attn.%s_proj.weight" % c].T).view(T, -1, D) for c in "qkv")
        a = _attend(_turn_halves(q, cs), _turn_halves(k, cs), v, lambda s, _: _softmax_weights(s * D ** -0.5, ok))
        x = x + a @ w[p + "self_attn.o_proj.weight"].T
        n = _rms(x, w[p + "post_attention_layernorm.weight"], eps)
        x = x + (_silu(n @ w[p + "mlp.gate_proj.weight"].T) * (n @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return lambda rows: _rms(x[rows], w["model.norm.weight"], eps) @ w["model.embed_tokens.weight"].T


def _livovik(cfg, w, ids):
    eps, alpha, T = cfg["norm"]["eps"], cfg["postln_alpha"], len(ids)
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        cs, ok = _angles(T, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"]), _seen(T, block=m["mask"]["size"])
        q, k, v = ((x @ w[p + "mix." + c].T).view(T, -1, m["dim"]) for c in "qkv")
        q, k = _turn_halves(_rms(q, w[p + "mix.q.norm"], eps), cs), _turn_halves(_rms(k, w[p + "mix.k.norm"], eps), cs)
        a = _attend(q, k, v, lambda s, h: _softmax_weights(s * m["scale"], ok, w[p + "mix.sink"][h]))
        a = (a.view(T, m["heads"], -1) * torch.sigmoid(x @ w[p + "mix.g"].T)[:, :, None]).reshape(T, -1)
        x = _rms(alpha * x + a @ w[p + "mix.o"].T, w[p + "norm1"], eps)
        x = _rms(alpha * x + torch.relu(x @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T, w[p + "norm2"], eps)
    return lambda rows: _rms(x[rows], w["final.norm"], eps) @ w["head"].T


def _state_space(n, w, p, m, eps):
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    I, T = H * P, n.shape[0]
    z, xbc, dt = (n @ w[p + "in"].T).split([I, I + 2 * G * N, H], 1)
    xbc = _silu(_conv(xbc, w[p + "conv"], w[p + "conv.b"]))
    x = xbc[:, :I].view(T, H, P)
    B, C = (xbc[:, I + i * G * N: I + (i + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"], threshold=60)
    a = torch.exp(-torch.exp(w[p + "A_log"]) * dt)
    S, y = torch.zeros(H, N, P, dtype=F64, device=DEVICE), torch.empty_like(x)
    for t in range(T):
        S = a[t][:, None, None] * S + dt[t][:, None, None] * B[t][:, :, None] * x[t][:, None]
        y[t] = (C[t][:, None] @ S)[:, 0]
    y = (y + w[p + "D"][:, None] * x).reshape(T, I) * _silu(z)
    return (_rms(y.view(T, m["norm_groups"], -1), None, eps).reshape(T, I) * w[p + "norm"]) @ w[p + "o"].T


def _mixed_heads(n, w, p, m, eps):
    T, H, G = n.shape[0], m["heads"], m["kv_heads"]
    q, k, v = ((n @ w[p + c].T + w[p + c + ".b"]).view(T, -1, m["dim"]) for c in "qkv")
    k, v = k.repeat_interleave(H // G, 1), _rms(v, None, eps).repeat_interleave(H // G, 1)
    sink = torch.zeros(H, dtype=F64, device=DEVICE)
    s = _softmax_weights(torch.einsum("ihd,jhd->hij", q, k) * m["scale"], _seen(T, window=m["mask"]["size"]), sink)
    s = (w[p + "talk"] @ s.view(H, T * T)).view(H, T, T)
    return torch.einsum("hij,jhd->ihd", s, v).reshape(T, -1) @ w[p + "o"].T


def _bazulorn(cfg, w, ids):
    eps = cfg["norm"]["eps"]
    x = _rms(w["embed"][ids], w["embed.norm"], eps)
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        n = _rms(x, w[p + "norm1"], eps)
        if layer["type"] == "parallel":
            y = 0.5 * (_rms(_mixed_heads(n, w, p + "mix.left.", m["left"], eps), w[p + "mix.left.out"], eps) +
                       _rms(_state_space(n, w, p + "mix.right.", m["right"], eps), w[p + "mix.right.out"], eps))
        else:
            y = _delta_mixer(n, w, p + "mix.", m, eps, True)
        x = x + y + (_gelu_tanh(n @ w[p + "mlp.gate"].T) * (n @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return lambda rows: _rms(x[rows], w["final.norm"], eps) @ w["embed"].T


def _purozen(cfg, w, ids):
    eps, T, first = cfg["norm"]["eps"], len(ids), None
    norm = lambda x, name: _rms(x, 1.0 + w[name], eps)
    gate = lambda n, name: torch.sigmoid(n @ w[name].T + w[name + ".b"])
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        n, a = norm(x, p + "norm1"), p + "mix."
        if layer["type"] == "parallel":
            left, ok = m["left"], _seen(T)
            q, k, v = ((n @ w[a + "left." + c].T).view(T, -1, left["dim"]) for c in "qkv")
            l = _attend(q, k, v, lambda s, h: torch.sigmoid(s * left["scale"] + w[a + "left.pb"][h, None, None]) * ok)
            z = torch.sigmoid(n @ w[a + "right.z"].T + w[a + "right.z.b"])
            u = n @ w[a + "right.x"].T + w[a + "right.x.b"]
            c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            S, rows = torch.zeros(z.shape[1], dtype=F64, device=DEVICE), torch.empty_like(z)
            for t in range(T):
                S = torch.lerp(S, c[t], z[t])
                rows[t] = S
            r = (rows * _silu(n @ w[a + "right.g"].T)) @ w[a + "right.o"].T
            y = m["left_scale"] * (l @ w[a + "left.o"].T) + m["right_scale"] * r
        elif layer["type"] == "attention":
            cs, ok = _angles(T, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"]), _seen(T, m["mask"]["size"], m["mask"]["keep_first"])
            q, k, v = ((n @ w[a + c].T).view(T, -1, m["dim"]) for c in "qkv")
            q, k = _rms(_turn_halves(q, cs), None, eps), _rms(_turn_halves(k, cs), None, eps)
            if first is None:
                first = v
            else:
                lam = w[a + "vmix"]
                v = (1 - lam) * v + lam * first
            y = _attend(q, k, v, lambda s, _: _softmax_weights(s * m["scale"], ok)) @ w[a + "o"].T
        else:
            c = _rms(n @ w[a + "dkv"].T, w[a + "dkv.norm"], eps)
            q, k, v = ((b @ w[a + name].T).view(T, m["heads"], -1) for b, name in ((n, "q"), (c, "uk"), (c, "uv")))
            y = _attend(q, k, v, lambda s, _: _softmax_weights(s * m["scale"], _seen(T))) @ w[a + "o"].T
        x = x + gate(n, p + "rg1") * y
        n = norm(x, p + "norm2")
        x = x + gate(n, p + "rg2") * (_gelu_tanh(n @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T)
    return lambda rows: norm(x[rows], "final.norm") @ w["embed"].T


def _danonex(cfg, w, ids):
    eps, mult, T = cfg["norm"]["eps"], cfg["residual_mult"], len(ids)
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        a = p + "mix."
        if layer["type"] == "attention":
            cs, ok = _angles(T, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"]), _seen(T)
            q, k = (_rms(x @ w[a + c].T, w[a + c + ".norm"], eps).view(T, -1, m["dim"]) for c in "qk")
            v = (x @ w[a + "v"].T).view(T, -1, m["vdim"])
            cap = m["softcap"]
            y = _attend(_turn_pairs(q, cs), _turn_pairs(k, cs), v, lambda s, h: _softmax_weights(
                cap * torch.tanh(s * m["scale"] / cap), ok, w[a + "sink"][h])) @ w[a + "o"].T
        else:
            y = _delta_mixer(x, w, a, m, eps, False)
        x = x + mult * _rms(y, w[p + "norm1"], eps)
        x = x + mult * _rms(_gelu_erf(x @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T, w[p + "norm2"], eps)
    return lambda rows: _rms(x[rows], w["final.norm"], eps) @ w["embed"].T * cfg["logit_scale"]


def _time_mixing(h, w, p, m, eps):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    x = {s: h + (before - h) * w[p + "mu." + s] for s in "rkvgw"}
    r, k, v = ((x[s] @ w[p + s].T).view(T, H, d) for s in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(x["w"] @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"])).view(T, H, d)
    u = w[p + "u"][:, :, None]
    S, o = torch.zeros(H, d, d, dtype=F64, device=DEVICE), torch.empty_like(v)
    for t in range(T):
        kv = k[t][:, :, None] * v[t][:, None]
        o[t] = (r[t][:, None] @ (S + u * kv))[:, 0]
        S = decay[t][:, :, None] * S + kv
    o = _rms(o, None, eps).reshape(T, H * d) * w[p + "norm"]
    return (o * _silu(x["g"] @ w[p + "g"].T)) @ w[p + "o"].T


def _query_latents(h, w, p, m, eps):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    cs = _angles(T, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])
    q = (_rms(h @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).view(T, H, -1)
    c, r = (h @ w[p + "dkv"].T).split([m["kv_rank"], m["rot_dim"]], 1)
    c = _rms(c, w[p + "dkv.norm"], eps)
    r = _turn_pairs(r[:, None], cs).expand(T, H, m["rot_dim"])
    q = torch.cat([q[..., :d], _turn_pairs(q[..., d:], cs)], -1)
    k = torch.cat([(c @ w[p + "uk"].T).view(T, H, d), r], -1)
    o = _attend(q, k, (c @ w[p + "uv"].T).view(T, H, -1), lambda s, _: _softmax_weights(s * m["scale"], _seen(T)))
    return (o * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def _zufotar(cfg, w, ids):
    eps = cfg["norm"]["eps"]
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p = "l%d." % i
        mixer = _time_mixing if layer["type"] == "wkv" else _query_latents
        y = mixer(_rms(x, w[p + "norm1"], eps), w, p + "mix.", layer["mixer"], eps)
        x = x + y + _gelu_erf(_rms(x, w[p + "norm2"], eps) @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T
    cap = cfg["logit_softcap"]
    return lambda rows: cap * torch.tanh(_rms(x[rows], w["final.norm"], eps) @ w["embed"].T / cap)


def exact(case, seed):
    contexts, decoded, prompts = _inputs(case, seed)
    if sum(map(len, contexts + prompts)) > (150000 if case["model"] == "llama" else 40000):     # over some twenty seconds
        return None
    cfg = config(case["model"], case["width"])
    w = _weights(cfg, seed)
    forward = {"llama": _llama, "livovik": _livovik, "bazulorn": _bazulorn, "purozen": _purozen, "danonex": _danonex,
               "zufotar": _zufotar}[case["model"]]
    steps = _portions(case)
    ids = lambda tokens: torch.tensor(tokens, device=DEVICE)
    of_decoding = [forward(cfg, w, ids(c + d[: len(steps)]))([len(c) + k for k in range(len(steps))]) for c, d in zip(contexts, decoded)]
    of_prompts = [forward(cfg, w, ids(p))([len(p) - 1]) for p in prompts]
    out = []
    for k, step in enumerate(steps):
        rows = [x[k: k + 1] for x in of_decoding] + [of_prompts[p] for p, _, b in step if b == len(prompts[p])]
        if rows:
            out.append(torch.cat(rows))
    return out
