"""The work that users of this repository have it do, through its public entry points.

Two libraries, each as its users' programs call it:

  the calm engine (calm_b200.lib.DeviceModel over the calm C boundary), one sequence of a Llama-shaped model
    kind "token"    forward(token, pos): one decode step against a cache of `pos` positions, logits back on the host
    kind "prompt"   prefill(all tokens but the last) and forward(the last one): a prompt up to its first logits
  the layer-list runtime (calm_b200.seqlib.SeqDeviceModel through the families' loaders), batches of sequences
    kind "ingest"   open, one step with a whole prompt per sequence, logits of each last token, close
    kind "generate" open, a prompt per sequence, `steps` decode steps (the argmax of every step is read, as a greedy
                    host does; the tokens fed are given, so that two implementations see the same ones), the logits of the
                    last step, close

Shapes are those of calm_b200.modelgen.SPECS and calm_b200.seqbench.SIZES.  The calm engine holds one model per process, as its
boundary says, and a program keeps its weights over all calls: prepare() builds a case's model once and keeps it until another case
asks for another model.  What the seed makes is the input: tokens, and for "generate" the prompts too."""
from __future__ import annotations

import math
import os

os.environ.setdefault("CALM_B200_QUIET", "1")

import numpy as np
import torch

from calm_b200 import bovinex, lib, modelgen, seqbench, vimulorn

FILL_SEED = 11  # of the cache contents before a decode step (calm_b200_fill_kv)


# --------------------------------------------------------------------------- the cases

def _engine(name, kind, spec, layers=None, **more):
    s = modelgen.SPECS[spec]
    c = {"name": name, "kind": kind, "dtype": s.dtype, "dim": s.dim, "hidden": s.hidden_dim, "layers": layers or s.n_layers, "heads": s.n_heads, "kv_heads": s.n_kv_heads,
         "head_dim": s.head_dim, "vocab": s.vocab_size, "theta": float(s.rope_theta), "eps": float(s.norm_eps), "bias": s.qkv_bias, "tied": s.tied,
         "experts": s.n_experts, "active": s.n_experts_active, "kvbits": 16}
    c.update(more)
    return c


def _seq(name, kind, family, size, blocks, **more):
    z = seqbench.SIZES[size]
    c = {"name": name, "kind": kind, "family": family, "blocks": blocks, **{k: z[k] for k in ("width", "ff", "heads", "dim", "kv_heads", "kv_rank", "q_rank", "window", "vocab")}}
    c.update(more)
    return c


def listed():
    return [
        # a small model on a short context: the latency of the launches of one token
        _engine("token 0.5b fp16 ctx 131", "token", "qwen2-0.5b-fp16", pos=131),
        # the headline: decode of a Llama-3-8B shape in fp8 at the end of a 4096-token context
        _engine("token 8b fp8 ctx 4095", "token", "llama3-8b-fp8", pos=4095),
        # the same model early in a conversation, fp16 weights, e5m2 cache
        _engine("token 8b fp16 kv8 ctx 1000", "token", "llama3-8b-fp16", layers=16, pos=1000, kvbits=8),
        # 4-bit groups: the format chosen to fit small memory
        _engine("token 7b gf4 ctx 2049", "token", "mistral-7b-gf4", pos=2049),
        # routed experts, two of eight read per token
        _engine("token 8x7b fp8 ctx 777", "token", "mixtral-8x7b-fp8", layers=8, pos=777),
        # a long prompt, a question with some context, a short question
        _engine("prompt 8b fp8 2047", "prompt", "llama3-8b-fp8", n=2047),
        _engine("prompt 7b gf4 333", "prompt", "mistral-7b-gf4", n=333),
        _engine("prompt 0.5b fp16 61", "prompt", "qwen2-0.5b-fp16", n=61),
        # layer-list models: a document into an attention / linear-attention model and into a latent / delta-rule / windowed one
        _seq("ingest bovinex 2048", "ingest", "bovinex", "w2048", 1, batch=1, prompt=2048),
        _seq("ingest vimulorn 3x700", "ingest", "vimulorn", "w2048", 1, batch=3, prompt=700),
        # chats: one user, and sixteen at once
        _seq("generate vimulorn 1x300", "generate", "vimulorn", "w1024", 2, batch=1, prompt=300, steps=64),
        _seq("generate bovinex 16x130", "generate", "bovinex", "w2048", 1, batch=16, prompt=130, steps=48),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["token", "token", "token", "prompt", "prompt", "ingest", "generate"])
    if kind in ("token", "prompt"):
        spec = rng.choice(["qwen2-0.5b-fp16", "llama3-8b-fp8", "mistral-7b-gf4", "llama3-8b-fp16", "mixtral-8x7b-fp8" if kind == "token" else "llama3-8b-gf4"])
        c = _engine(None, kind, spec, layers=rng.choice([4, 6, 8, 12]), kvbits=rng.choice([16, 16, 8]))
        if c["experts"]:
            c["layers"] = rng.choice([2, 3, 4])
        elif rng.random() < 0.5:  # widths between the named shapes
            c["heads"] = 4 * rng.choice([3, 4, 6, 8])
            c["kv_heads"] = c["heads"] // 4
            c["head_dim"] = 128 if c["heads"] == 12 else rng.choice([64, 128])
            c["dim"] = c["heads"] * c["head_dim"]
            c["hidden"] = 128 * round(c["dim"] * rng.uniform(2.5, 4.0) / 128)
            c["bias"] = c["tied"] = False
        if kind == "token":
            c["pos"] = _log(rng, 8, 4095)
        else:
            c["n"] = _log(rng, 9, 2047)
    else:
        c = _seq(None, kind, rng.choice(["bovinex", "vimulorn"]), rng.choice(["w1024", "w2048"]), 1)
        c["batch"] = _log(rng, 1, 16)
        if kind == "ingest":
            c["prompt"] = _log(rng, 33, 2048 // c["batch"])
        else:
            c["prompt"], c["steps"] = _log(rng, 17, 400 if c["batch"] < 4 else 130), rng.randint(16, 64)
    del c["name"]
    return c


# --------------------------------------------------------------------------- models

class _Kept:
    """The one model in memory, by what determines it."""

    key = model = data = None


def _spec(c):
    return modelgen.ModelSpec("case", c["dim"], c["hidden"], c["layers"], c["heads"], c["kv_heads"], c["head_dim"], c["vocab"], c["dtype"], rope_theta=c["theta"], norm_eps=c["eps"],
                              n_experts=c["experts"], n_experts_active=c["active"], qkv_bias=c["bias"], tied=c["tied"])


def _config(c):
    cfg = (seqbench.bovinex_config if c["family"] == "bovinex" else seqbench.vimulorn_config)(c)
    for lc in cfg["layers"]:
        if lc["mlp"]["kind"] == "moe":  # in 16 bits a rounding can change which experts a token goes to: dense units here, the engine's case has experts
            lc["mlp"] = {"ff": c["ff"], "kind": "dense"}
    return cfg


def _seq_tensors(c):
    """bf16 weights with the distributions of the families' own synthetic checkpoints, made on the GPU."""
    cfg = _config(c)
    g = torch.Generator(device="cuda").manual_seed(5)
    out = {}
    for name, shape in (bovinex if c["family"] == "bovinex" else vimulorn).tensor_shapes(cfg).items():
        leaf = name.split(".")[-1]
        t = torch.randn(shape, generator=g, device="cuda")
        if leaf == "alpha":
            t = 0.75 + 0.05 * t
        elif name.endswith("a2.b"):
            t = 1.5 + 1.5 * t
        elif c["family"] == "bovinex" and (leaf == "norm1" or name == "final.norm"):
            t = 0.2 * t
        elif leaf.startswith("norm") or leaf == "norm":
            t = 1.0 + 0.1 * t
        elif name.endswith(".b"):
            t = (0.05 if "norm" in name else 0.3) * t
        elif leaf == "conv":
            t = t / math.sqrt(shape[1])
        elif leaf == "A_log":
            t = (0.5 + 2.0 * torch.sigmoid(t)).log()
        elif leaf == "embed":
            t = t / float((cfg.get("embedding") or {}).get("scale", 1.0))
        elif leaf not in ("dt_bias", "sink"):
            t = t * (1.3 / math.sqrt(shape[-1]))
        out[name] = t.to(torch.bfloat16)
    return cfg, out


def _weights(c):
    return modelgen.generate(_spec(c), seed=3, device="cuda")


def _model(c):
    engine = c["kind"] in ("token", "prompt")
    key = tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "kind", "n", "prompt", "steps", "batch") and not (engine and k == "pos")))
    at = c.get("pos")  # how far the cache is filled
    if _Kept.key != (engine, key):
        if _Kept.model is not None:
            _Kept.model.close()
        _Kept.key = _Kept.model = _Kept.data = None
        torch.cuda.empty_cache()
        if engine:
            _Kept.data = _weights(c)
            torch.cuda.synchronize()
            _Kept.model = lib.DeviceModel(_spec(c), _Kept.data, seq_len=4096, kvbits=c["kvbits"])
        else:
            cfg, tensors = _seq_tensors(c)
            tensors = {k: v.cpu() for k, v in tensors.items()}
            _Kept.model = (bovinex if c["family"] == "bovinex" else vimulorn).from_tensors(cfg, tensors, "bfloat16", max_tokens=8192, max_seqs=16)
        _Kept.key = (engine, key)
    if at is not None:
        _Kept.model.fill_kv(at, FILL_SEED)
    return _Kept.model


def _tokens(c, seed, rows, n):
    return np.random.default_rng([seed, rows, n]).integers(3, c["vocab"], (rows, n)).astype(np.int32)


def _inputs(c, seed):
    if c["kind"] == "token":
        return int(_tokens(c, seed, 1, 8)[0, seed % 8])
    if c["kind"] == "prompt":
        return _tokens(c, seed, 1, c["n"])[0]
    # prompts of several lengths: the one asked for, and shorter ones
    lens = [max(1, c["prompt"] - (7 * i) % max(1, c["prompt"] // 2)) for i in range(c["batch"])]
    rows = [list(map(int, _tokens(c, seed + 1000 * i, 1, n)[0])) for i, n in enumerate(lens)]
    return rows, _tokens(c, seed + 77, c.get("steps", 0) or 1, c["batch"])


def prepare(case, seed):
    return {"case": case, "model": _model(case), "inputs": _inputs(case, seed)}


def run(state):
    c, m, given = state["case"], state["model"], state["inputs"]
    if c["kind"] == "token":
        return m.forward(given, c["pos"])
    if c["kind"] == "prompt":
        m.prefill(given[:-1], 0)
        return m.forward(int(given[-1]), c["n"] - 1)
    prompts, then = given
    slots = [m.open() for _ in prompts]
    ends = np.cumsum([len(p) for p in prompts]) - 1
    if c["kind"] == "ingest":
        out = m.step(slots, prompts, ends)
    else:
        m.step(slots, prompts, ends, fetch=False)
        every = list(range(len(slots)))
        for s in range(c["steps"]):
            m.argmax(len(slots))
            out = m.step(slots, [[int(t)] for t in then[s]], every, fetch=s + 1 == c["steps"])
    for s in slots:
        m.close_seq(s)
    return out


# --------------------------------------------------------------------------- work

def work(case):
    """What a pass cannot do without: every weight that it needs once, the cache once, two operations per weight and token."""
    c = case
    if c["kind"] in ("token", "prompt"):
        s = _spec(c)
        n = 1 if c["kind"] == "token" else c["n"]
        wbytes = modelgen.algorithmic_bytes(s)
        per_token = c["layers"] * (c["dim"] * (2 * s.q_dim + 2 * s.kv_dim) + 3 * c["dim"] * c["hidden"] * (c["active"] or 1))
        ctx = c["pos"] + 1 if c["kind"] == "token" else n
        kv = modelgen.kv_bytes(s, ctx - 1, 4096, c["kvbits"])
        attn = 4 * c["layers"] * s.q_dim * (ctx if n == 1 else n * (n + 1) // 2)
        return {"bytes": wbytes + kv + 4 * c["vocab"], "flops": 2 * n * per_token + attn + 2 * c["dim"] * c["vocab"]}
    shapes = (bovinex if c["family"] == "bovinex" else vimulorn).tensor_shapes(_config(c))
    lens = [len(p) for p in _inputs(c, 0)[0]]
    steps = c.get("steps", 0)
    mats = sum(int(np.prod(v)) for k, v in shapes.items() if k not in ("embed", "head"))
    head = int(np.prod(shapes["head"]))
    toks = sum(lens)
    nbytes = 2 * mats + 2 * head + 4 * c["batch"] * c["vocab"] + steps * (2 * mats + 2 * head)
    flops = 2 * mats * (toks + steps * c["batch"]) + 2 * head * c["batch"] * (1 + steps)
    for lc in _config(c)["layers"]:
        mx = lc["mixer"]
        w = (mx.get("mask") or {}).get("size", 1 << 30)
        if lc["type"] in ("attention", "latent_attention"):
            keys = sum(min(i + 1, w) for n in lens for i in range(n + steps))
            flops += 4 * mx["heads"] * mx["dim"] * keys
            row = mx["kv_rank"] if "kv_rank" in mx else 2 * mx["kv_heads"] * mx["dim"]
            nbytes += 4 * row * (toks + sum(min(n + s + 1, w) for n in lens for s in range(steps)))
        else:
            flops += 4 * mx["heads"] * mx["dim"] * mx["vdim"] * (toks + steps * c["batch"])
            nbytes += 8 * mx["heads"] * mx["dim"] * mx["vdim"] * c["batch"] * (1 + steps)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the distance from the 64-bit statement that was seen over listed and drawn cases.  Engine: sums and activations in 32
    bits, cache entries rounded to fp16 (a rounding that falls the other way travels on): 1.8e-4 for a token, 8.3e-4 for a prompt.  Layer-list
    models: products of bf16 inputs, 4e-3 to 1e-2."""
    return {"rel": {"token": 7e-4, "prompt": 3.3e-3}.get(case["kind"], 3e-2)}


# --------------------------------------------------------------------------- plain statements in 64 bits

F = torch.float64


def _plain_weight(t, dtype):
    if dtype == "fp16":
        return t.to(F)
    if dtype == "fp8":
        return t.view(torch.float8_e5m2).to(torch.float32).to(F)
    w = t.to(torch.int64) & 0xFFFFFFFF
    scale = (w & 255).to(torch.uint8).view(torch.float8_e5m2).to(torch.float32).to(F) / -4.0
    codes = (w[..., None] >> (8 + 3 * torch.arange(8, device=w.device))) & 7
    return ((codes - 4).to(F) * scale[..., None]).flatten(-2)


def _shr(z, n):  # logical shift of a 64-bit pattern
    return (z >> n) & ((1 << (64 - n)) - 1)


def _cache_fill(c, layer, npos):
    """The cache contents that calm_b200_fill_kv(npos, FILL_SEED) leaves for one layer: (k, v) [kv_heads, npos, head_dim]."""
    per = c["kv_heads"] * npos * c["head_dim"]
    u64 = lambda v: v - (1 << 64) if v >= 1 << 63 else v  # noqa: E731
    i = torch.arange(layer * per, (layer + 1) * per, device="cuda")
    z = (i + 1) * u64(0x9E3779B97F4A7C15) + FILL_SEED
    z = (z ^ _shr(z, 30)) * u64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * u64(0x94D049BB133111EB)
    z = z ^ _shr(z, 31)
    shape = (c["kv_heads"], npos, c["head_dim"])
    both = [(((x & 0xFFFFFF).to(F) / 16777216.0 - 0.5) * 2.0).reshape(shape) for x in (z, _shr(z, 24))]
    return [_cached(x, c) for x in both]


def _cached(x, c):
    """Rounded to the cache's element type."""
    return x.to(torch.float32).to(torch.float16 if c["kvbits"] == 16 else torch.float8_e5m2).to(torch.float32).to(F)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _exact_engine(c, seed):
    W = _weights(c)
    dt = c["dtype"]
    mat = lambda name: _plain_weight(W[name], dt)  # noqa: E731
    toks = _inputs(c, seed)
    toks = torch.as_tensor(np.atleast_1d(np.asarray(toks, np.int64)), device="cuda")
    pos = torch.arange(len(toks), device="cuda") + (c["pos"] if c["kind"] == "token" else 0)
    H, G, D = c["heads"], c["kv_heads"], c["head_dim"]
    freq = torch.tensor([c["theta"] ** (-2.0 * i / D) for i in range(D // 2)], dtype=F, device="cuda")
    ang = pos[:, None].to(F) * freq
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def turn(v):  # [T, heads, D], channels 2i and 2i + 1
        a, b = v[..., 0::2], v[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)

    x = _plain_weight(W["model.embed.weight"][toks], dt)
    for l in range(c["layers"]):
        p = f"model.layers.{l}."
        h = _rms(x, W[p + "attn.norm.weight"].to(F), c["eps"])
        qkv = [h @ mat(p + f"attn.w{n}.weight").T for n in "qkv"]
        if c["bias"]:
            b = W[p + "attn.wqkv.bias"].to(F)
            qkv = [y + z for y, z in zip(qkv, b.split([H * D, G * D, G * D]))]
        q, k = turn(qkv[0].reshape(-1, H, D)), _cached(turn(qkv[1].reshape(-1, G, D)), c)
        v = _cached(qkv[2].reshape(-1, G, D), c)
        k, v = k.transpose(0, 1), v.transpose(0, 1)
        if c["kind"] == "token" and c["pos"]:
            k0, v0 = _cache_fill(c, l, c["pos"])
            k, v = torch.cat([k0, k], 1), torch.cat([v0, v], 1)
        att = torch.empty_like(q)
        seen = torch.arange(k.shape[1], device="cuda")[None, :] <= pos[:, None]
        for hd in range(H):
            s = (q[:, hd] @ k[hd * G // H].T) / math.sqrt(D)
            att[:, hd] = s.masked_fill(~seen, -math.inf).softmax(-1) @ v[hd * G // H]
        x = x + att.flatten(1) @ mat(p + "attn.wo.weight").T
        h = _rms(x, W[p + "mlp.norm.weight"].to(F), c["eps"])
        if c["experts"]:
            z = h @ _plain_weight(W[p + "moegate.weight"], dt).T
            best, which = z.softmax(-1).topk(c["active"], -1)
            best = best / best.sum(-1, keepdim=True)
            units = [(int(e), best[0, j]) for j, e in enumerate(which[0])]  # one token
        else:
            units = [(None, 1.0)]
        y = 0
        for e, weight in units:
            w1, w2, w3 = (_plain_weight(W[p + f"mlp.w{n}.weight"] if e is None else W[p + f"mlp.w{n}.weight"][e], dt) for n in (1, 2, 3))
            y = y + weight * ((torch.nn.functional.silu(h @ w1.T) * (h @ w3.T)) @ w2.T)
        x = x + y
    last = _rms(x[-1], W["model.norm.weight"].to(F), c["eps"])
    name = "model.embed.weight" if c["tied"] else "model.output.weight"
    return torch.cat([_plain_weight(W[name][r:r + 8192], dt) @ last for r in range(0, c["vocab"], 8192)])


def _attend(q, k, v, scale, window=None, keep=0, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv], causal."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=q.device)
    far = i[:, None] - i[None, :]
    seen = far >= 0
    if window:
        seen &= (far < window) | (i[None, :] < keep)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(s.softmax(-1)[:, :T] @ v[:, h * G // H])
    return torch.stack(out, 1)


def _conv(u, w):
    taps = w.shape[1]
    pad = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u], 0)
    return sum(pad[j:j + u.shape[0]] * w[:, j] for j in range(taps))


def _exact_bovinex(cfg, P, toks):
    eps = cfg["norm"]["eps"]
    x = P["embed"][toks] * cfg["embedding"]["scale"]
    T = len(toks)
    for i, lc in enumerate(cfg["layers"]):
        m, mx = f"l{i}.mix.", lc["mixer"]
        H, D, Dv = mx["heads"], mx["dim"], mx["vdim"]
        h = _rms(x, 1.0 + P[f"l{i}.norm1"], eps)
        g = h @ P[m + "g"].T
        if lc["type"] == "attention":
            G, rot = mx["kv_heads"], mx["rot"]
            q = _rms(h @ P[m + "q"].T + P[m + "q.b"], P[m + "q.norm"], eps).reshape(T, H, D)
            k = _rms(h @ P[m + "k"].T + P[m + "k.b"], P[m + "k.norm"], eps).reshape(T, G, D)
            v = (h @ P[m + "v"].T + P[m + "v.b"]).reshape(T, G, Dv)
            n, sc = rot["dims"], rot["scaling"]
            f = torch.tensor([rot["base"] ** (-2.0 * j / n) for j in range(n // 2)], dtype=F, device=x.device)
            at = lambda turns: n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))  # noqa: E731
            lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
            ramp = ((torch.arange(n // 2, device=x.device, dtype=F) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
            f = f / sc["factor"] * ramp + f * (1 - ramp)
            ang = torch.arange(T, device=x.device, dtype=F)[:, None] * f
            mag = 0.1 * math.log(sc["factor"]) + 1.0
            cs, sn = (ang.cos() * mag)[:, None], (ang.sin() * mag)[:, None]

            def turn(u):
                a, b = u[..., :n // 2], u[..., n // 2:n]
                return torch.cat([a * cs - b * sn, b * cs + a * sn, u[..., n:]], -1)

            o = _attend(turn(q), turn(k), v, mx["scale"], mx["mask"]["size"], mx["mask"]["keep_first"]).flatten(1) * torch.sigmoid(g)
        else:
            q = (h @ P[m + "q"].T).reshape(T, H, D) * D ** -0.5
            k = (h @ P[m + "k"].T).reshape(T, H, D)
            v = (h @ P[m + "v"].T).reshape(T, H, Dv)
            a = torch.exp(torch.nn.functional.logsigmoid((h @ P[m + "a1"].T) @ P[m + "a2"].T + P[m + "a2.b"]) / mx["tau"]).reshape(T, H, D)
            S, o = x.new_zeros(H, D, Dv), x.new_empty(T, H, Dv)
            for t in range(T):
                S = a[t, :, :, None] * S + k[t, :, :, None] * v[t, :, None, :]
                o[t] = (q[t, :, None, :] @ S)[:, 0]
            o = _rms(o, P[m + "norm"], eps).flatten(1) * torch.nn.functional.silu(g)
        x = x + o @ P[m + "o"].T + torch.relu(h @ P[f"l{i}.mlp.up"].T) ** 2 @ P[f"l{i}.mlp.down"].T
    return _rms(x[-1], 1.0 + P["final.norm"], eps) @ P["head"].T


def _exact_vimulorn(cfg, P, toks):
    eps = cfg["norm"]["eps"]
    dyt = lambda y, n: torch.tanh(P[n + ".alpha"] * y) * P[n] + P[n + ".b"]  # noqa: E731
    one = torch.ones((), dtype=F, device="cuda")
    x = P["embed"][toks]
    T = len(toks)
    silu = torch.nn.functional.silu
    for i, lc in enumerate(cfg["layers"]):
        m, mx = f"l{i}.mix.", lc["mixer"]
        H, D, Dv = mx["heads"], mx["dim"], mx["vdim"]
        h = dyt(x, f"l{i}.norm1")
        if lc["type"] == "latent_attention":
            q = (_rms(h @ P[m + "dq"].T, P[m + "dq.norm"], eps) @ P[m + "uq"].T).reshape(T, H, D)
            lat = _rms(h @ P[m + "dkv"].T, P[m + "dkv.norm"], eps)
            o = _attend(q, (lat @ P[m + "uk"].T).reshape(T, H, D), (lat @ P[m + "uv"].T).reshape(T, H, Dv), mx["scale"]) * torch.sigmoid(h @ P[m + "g"].T)[:, :, None]
        elif lc["type"] == "channel_delta":
            G = mx["kv_heads"]
            q, k = (silu(_conv(h @ P[m + n].T, P[m + n + ".conv"])).reshape(T, G, D) for n in "qk")
            v = silu(_conv(h @ P[m + "v"].T, P[m + "v.conv"])).reshape(T, H, Dv)
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5).repeat_interleave(H // G, 1)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
            beta = torch.sigmoid(h @ P[m + "b"].T)
            dt = torch.nn.functional.softplus((h @ P[m + "a1"].T) @ P[m + "a2"].T + P[m + "dt_bias"], threshold=200).reshape(T, H, D)
            a = torch.exp(-torch.exp(P[m + "A_log"])[None, :, None] * dt)
            S, o = x.new_zeros(H, D, Dv), x.new_empty(T, H, Dv)
            for t in range(T):
                S = a[t, :, :, None] * S
                u = beta[t, :, None] * (v[t] - (k[t, :, None, :] @ S)[:, 0])
                S = S + k[t, :, :, None] * u[:, None, :]
                o[t] = (q[t, :, None, :] @ S)[:, 0]
            o = _rms(o, P[m + "norm"], eps) * torch.sigmoid((h @ P[m + "g1"].T) @ P[m + "g2"].T).reshape(T, H, Dv)
        else:
            G = mx["kv_heads"]
            q, k, v = (_conv(h @ P[m + n].T, P[m + n + ".conv"]).reshape(T, -1, d) for n, d in (("q", D), ("k", D), ("v", Dv)))
            o = _attend(_rms(q, one, eps), _rms(k, one, eps), v, mx["scale"], mx["mask"]["size"], sink=P[m + "sink"])
        x = x + dyt(o.flatten(1) @ P[m + "o"].T, f"l{i}.norm1b")
        h, lim = dyt(x, f"l{i}.norm2"), lc["mlp"]["limit"]
        gate, up = (h @ P[f"l{i}.mlp.gate"].T).clamp(max=lim), (h @ P[f"l{i}.mlp.up"].T).clamp(-lim, lim)
        x = x + dyt((gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ P[f"l{i}.mlp.down"].T, f"l{i}.norm2b")
    return dyt(x[-1], "final.norm") @ P["head"].T


def exact(case, seed):
    if case["kind"] in ("token", "prompt"):
        return _exact_engine(case, seed)
    cfg, P = _seq_tensors(case)
    P = {k: v.to(F) for k, v in P.items()}
    rows, then = _inputs(case, seed)
    plain = _exact_bovinex if case["family"] == "bovinex" else _exact_vimulorn
    if case["kind"] == "generate":
        rows = [r + [int(t) for t in then[:, i]] for i, r in enumerate(rows)]
    return torch.stack([plain(cfg, P, torch.as_tensor(r, device="cuda")) for r in rows])
