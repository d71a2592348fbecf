"""The work this framework is measured on: token loops and prompt passes through the public model API.

A case is one model shape, what it already has in its cache (`cached` prompt tokens, fed when the state is prepared) and
one pass of use: rewind to the cached prompt, feed `new` prompt tokens in one call, score `scored` given tokens one call
each (logits to the host, as a constrained decoder or an evaluation does), then let the device loop produce `steps` tokens
(greedy, top-k, full vocabulary, or several samples sharing the prompt).

Weights are the framework's own seeded synthetic ones.  The decoders whose loops return token ids have the scale
0.192 / sqrt(dim): the embedding keeps a share of the residual stream, as in a trained model, so the loops' choices rest on
clear winners and ids can be compared.  Configured decoders (norms behind every sublayer) are scored on given tokens.
"""
import math

import numpy as np
import torch

import rustane_b200 as R


# ------------------------------------------------------------------------------------------------ the cases
def dense(name, dim, hidden, heads, kv_heads, hd, layers, vocab, seq, dtype, cached, new=0, scored=0, steps=0, mode="greedy", samples=1,
          untied=False, activation=0):
    c = dict(family="dense", dim=dim, hidden=hidden, heads=heads, kv_heads=kv_heads, hd=hd, layers=layers, vocab=vocab, seq=seq, dtype=dtype,
             cached=cached, new=new, scored=scored, steps=steps, mode=mode, samples=samples, untied=untied, activation=activation)
    return dict(c, name=name) if name else c


def moe(name, dim, hidden, heads, layers, vocab, experts, top, shared, cached, new, scored, steps):
    c = dict(family="moe", dim=dim, hidden=hidden, heads=heads, layers=layers, vocab=vocab, seq=8192, experts=experts, top=top, shared=shared,
             latent=512, rope=64, nope=128, vdim=128, dtype="bf16", cached=cached, new=new, scored=scored, steps=steps, mode="greedy", samples=1)
    return dict(c, name=name) if name else c


def configured(name, family, pattern, dim, hidden, heads, kv_heads, layers, vocab, window, side, new, scored, cached=0):
    c = dict(family=family, pattern=pattern, dim=dim, hidden=hidden, heads=heads, kv_heads=kv_heads, layers=layers, vocab=vocab, seq=8192,
             window=window, side=side, dtype="bf16", cached=cached, new=new, scored=scored, steps=0, mode="greedy", samples=1)
    return dict(c, name=name) if name else c


def listed():
    five = (4096, 11008, 32, 32, 128, 26, 32000, 4096)  # the benchmark's 5B decoder
    return [
        # the smallest model and prompt, fp32: launches and latency
        dense("tiny_f32_tokens", 512, 1536, 8, 8, 64, 8, 8192, 512, "f32", cached=4, scored=2, steps=32),
        # a chat turn on a small model: a ragged suffix behind the cached conversation, then sampled tokens
        dense("600m_f16_turn_topk", 1536, 4096, 12, 12, 128, 24, 32000, 2048, "f16", cached=512, new=37, scored=1, steps=48, mode="topk"),
        # grouped queries, as most models of this size have them, in the middle of a long conversation (ragged length)
        dense("1b_bf16_grouped_tokens", 2048, 5632, 16, 4, 128, 24, 32000, 4096, "bf16", cached=1999, scored=1, steps=48),
        # the headline: batch-1 decode of the 5B model behind a 1024-token prompt
        dense("5b_bf16_tokens", *five, "bf16", cached=1024, scored=1, steps=32),
        # prompts of the 5B model: an ordinary one and the longest the model takes
        dense("5b_bf16_prompt_1024", *five, "bf16", cached=0, new=1024),
        dense("5b_bf16_prompt_4096", *five, "bf16", cached=0, new=4096),
        # the quantised models people run for speed
        dense("5b_fp8_tokens", *five, "fp8", cached=1024, scored=1, steps=32),
        dense("5b_int4_tokens", *five, "int4", cached=160, scored=1, steps=32),
        # eight samples of one prompt, the whole vocabulary sampled
        dense("5b_bf16_eight_samples", *five, "bf16", cached=1024, scored=1, steps=16, mode="samples", samples=8),
        # the mixture of experts behind latent attention
        moe("moe_latent_tokens", 2048, 1408, 16, 24, 32000, 64, 6, 2, cached=250, new=0, scored=1, steps=32),
        # configured decoders: a document read, then tokens scored one by one
        configured("dafidra_1b_read_and_score", "dafidra", "p", 2048, 5632, 16, 4, 24, 32000, 1024, 0, new=1500, scored=24),
        configured("kazodra_1b_read_and_score", "kazodra", "lssa", 2048, 5632, 16, 4, 24, 32000, 1024, 128, new=2048, scored=24),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["dense"] * 5 + ["prompt"] * 2 + ["moe", "dafidra", "kazodra"])
    vocab = int(_log(rng, 2000, 40000))
    if kind == "moe":
        return moe(None, 256 * rng.randint(4, 8), 128 * rng.randint(4, 11), rng.choice([8, 16]), rng.randint(4, 24), vocab, rng.choice([16, 32, 64]),
                   rng.choice([2, 4, 6]), rng.randint(1, 2), int(_log(rng, 20, 400)), 0, rng.randint(1, 3), rng.randint(8, 32))
    if kind in ("dafidra", "kazodra"):
        heads = rng.choice([8, 16, 16, 24])
        pattern = "p" if kind == "dafidra" else rng.choice(["lssa", "l", "s", "a", "sa"])
        return configured(None, kind, pattern, 128 * heads + rng.choice([0, 0, 64, 8]), 8 * int(_log(rng, 256, 704)), heads, rng.choice([2, 4, 8]),
                          rng.randint(2, 24), vocab, int(_log(rng, 64, 1024)), rng.choice([0, 96, 128]) if kind == "kazodra" else 0,
                          new=int(_log(rng, 24, 2048)), scored=rng.randint(1, 24))
    hd = rng.choice([64, 128, 128])
    dim = 64 * int(_log(rng, 8, 65))
    group = rng.choice([1, 1, 2, 4, 8])
    heads = max(group, dim // hd // group * group)
    hidden = 32 * int(dim * rng.uniform(2.0, 3.5) / 32)
    layers = rng.randint(2, 26)
    if kind == "prompt":
        cached = rng.choice([0, 0, int(_log(rng, 16, 1024))])
        return dense(None, dim, hidden, heads, heads // group, hd, layers, vocab, 4096, rng.choice(["bf16", "bf16", "f16", "fp8"]), cached,
                     new=int(_log(rng, 16, 3000)), activation=rng.choice([0, 0, 1]))
    mode = rng.choice(["greedy", "greedy", "topk", "fullvocab", "samples"])
    dtype = rng.choice(["f32", "f16", "f16", "bf16", "bf16", "bf16", "fp8", "fp8", "int4"])
    if mode == "samples":
        dtype = rng.choice(["f16", "bf16"])
    if mode in ("fullvocab", "samples"):
        dim = max(dim, 2048)
        heads = max(group, dim // hd // group * group)
        hidden = 32 * int(dim * rng.uniform(2.0, 3.0) / 32)
    if dtype == "f32" and dim > 2048:
        dim, hidden = dim // 2, hidden // 2 // 32 * 32
        heads = max(group, dim // hd // group * group)
    slow = dtype in ("f32", "int4")  # their prompts go one token at a time
    return dense(None, dim, hidden, heads, heads // group, hd, layers, vocab, 4096, dtype, int(_log(rng, 4, 200 if slow else 3500)),
                 new=rng.choice([0, 0, int(_log(rng, 2, 12 if slow else 200))]), scored=rng.randint(1, 2), steps=rng.randint(8, 32), mode=mode,
                 samples=rng.choice([2, 4, 8, 11, 16]) if mode == "samples" else 1, untied=False, activation=rng.choice([0, 0, 0, 1]))


# ------------------------------------------------------------------------------------------------ models
def dafidra_json(c):
    H = c["heads"] // 2
    layer = {"type": "parallel", "mlp": {"kind": "dense", "ff": c["hidden"]}, "mixer": {
        "left": {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": c["window"]},
                 "q_temp": {"coef": 0.1, "every": 4096}},
        "right": {"heads": H, "dim": 128, "vdim": 256, "gate_cap": 15.0}}}
    return {"architecture": "Dafidra", "width": c["dim"], "vocab": c["vocab"], "norm": {"eps": 1e-5}, "residual_mult": 0.5, "layers": [layer] * c["layers"]}


def kazodra_json(c):
    heads = c["heads"]
    mixers = {
        "a": ("attention", {"heads": heads, "kv_heads": c["kv_heads"], "dim": 64, "vdim": 128, "scale": 0.125, "diff": 0.5,
                            "rot": {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}}}),
        "l": ("latent_attention", {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                                   "rot": {"dims": 64, "base": 10000.0}, "mask": {"size": c["window"]}}),
        "s": ("lightning", {"heads": heads, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(2 + 8.0 * h / heads) for h in range(heads)]}),
    }
    layers = []
    for i in range(c["layers"]):
        kind, m = mixers[c["pattern"][i % len(c["pattern"])]]
        layers.append({"type": kind, "mixer": m, "mlp": {"kind": "dense", "ff": c["hidden"]}})
    cfg = {"architecture": "Kazodra", "width": c["dim"], "vocab": c["vocab"], "norm": {"eps": 1e-5}, "layers": layers}
    if c["side"]:
        cfg["token_side"] = {"dim": c["side"]}
    return cfg


def std_of(c):
    return 0.02 if c["family"] in ("dafidra", "kazodra") else 0.192 / math.sqrt(c["dim"])


def build(c, seed):
    seed += 1
    if c["family"] == "dense":
        cfg = R.Config(c["dim"], c["hidden"], c["heads"], c["hd"], c["seq"], c["layers"], c["vocab"], kv_heads=c["kv_heads"])
        return R.Model.synthetic(cfg, seed, std=std_of(c), untied_head=c["untied"], dtype=c["dtype"], activation=c["activation"], use_graph=True,
                                 max_samples=c["samples"])
    if c["family"] == "moe":
        cfg = R.MoeConfig(c["dim"], c["hidden"], c["heads"], c["seq"], c["layers"], c["vocab"], c["experts"], c["top"], c["shared"], c["latent"],
                          c["rope"], c["nope"], c["vdim"])
        return R.Model.moe_synthetic(cfg, seed, std=std_of(c), dtype=c["dtype"], use_graph=True)
    cfg = dafidra_json(c) if c["family"] == "dafidra" else kazodra_json(c)
    return R.Model.from_config(cfg, seed, std=std_of(c), max_tokens=c["seq"], dtype=c["dtype"], use_graph=True)


def tokens_of(c, seed):
    """Prompt in the cache, prompt of the pass, tokens to score, first tokens of the loop (one per sample), random states."""
    rng = np.random.default_rng([seed, 77])
    ids = [rng.integers(0, c["vocab"], n, dtype=np.int64).astype(np.uint32) for n in (c["cached"], c["new"], c["scored"], c["samples"])]
    return ids, rng.integers(1, 1 << 62, c["samples"], dtype=np.int64).astype(np.uint64)


def prepare(case, seed):
    (cached, new, scored, first), rng = tokens_of(case, seed)
    m = build(case, seed)
    if len(cached):
        m.prefill(cached, want_logits=False)
    return {"model": m, "case": case, "new": new, "scored": [int(t) for t in scored], "first": first, "rng": rng}


def run(state):
    m, c, out = state["model"], state["case"], {}
    m.set_len(c["cached"])
    if c["new"]:
        out["prompt_logits"] = m.prefill(state["new"])
    if c["scored"]:
        out["scored_logits"] = [m.decode_token_logits_from_id(t) for t in state["scored"]]
    if c["steps"]:
        first = int(state["first"][0])
        if c["mode"] == "greedy":
            out["ids"] = m.decode_steps_greedy(first, c["steps"])
        elif c["mode"] == "topk":
            out["ids"] = m.decode_steps_topk(first, c["steps"], 8, 0.5, int(state["rng"][0]))[0]
        elif c["mode"] == "fullvocab":
            out["ids"] = m.decode_steps_fullvocab(first, c["steps"], 0.3, int(state["rng"][0]))[0]
        else:
            out["ids"] = m.decode_steps_samples(state["first"], c["steps"], mode="fullvocab", temperature=0.3, rng_states=state["rng"])[0]
        out["ids"] = out["ids"].astype(np.int64)
    return out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _parts(c):
    """(weights a token multiplies with, of these the ones held as 16 or 32 bits whatever the type, elements cached per
    position and layer, multiply-adds per query-key pair and layer, layers that attend, window)."""
    D, L = c["dim"], c["layers"]
    head = c["vocab"] * D
    if c["family"] == "dense":
        Q, KV = c["heads"] * c["hd"], c["kv_heads"] * c["hd"]
        return L * (D * (2 * Q + 2 * KV) + 3 * D * c["hidden"]), head, 2 * KV, 2 * Q, L, 1 << 30
    if c["family"] == "moe":
        qh, w = c["nope"] + c["rope"], c["latent"] + c["rope"]
        attn = D * (c["heads"] * qh + w) + c["latent"] * c["heads"] * (c["nope"] + c["vdim"]) + c["heads"] * c["vdim"] * D
        return L * (attn + 3 * D * c["hidden"] * (c["top"] + c["shared"]) + D * c["experts"]), head, w, c["heads"] * (w + c["latent"]), L, 1 << 30
    if c["family"] == "dafidra":
        H, G = c["heads"], c["kv_heads"]
        rows = 128 * (H + 2 * G) + H + H // 2 * (2 * 128 + 2 * 256 + 2)
        return L * (D * (rows + H * 128 + H // 2 * 256) + 3 * D * c["hidden"]), head, 256 * G, 2 * H * 128, L, c["window"]
    w = kv = pairs = 0
    H, G = c["heads"], c["kv_heads"]
    for i in range(L):
        k = c["pattern"][i % len(c["pattern"])]
        if k == "l":
            w += D * (H * 192 + 576) + 512 * H * 256
            kv, pairs = kv + 576, pairs + H * (192 + 128)
        elif k == "s":
            w += D * H * 512
        else:
            w += D * (128 * (H + G) + 128 * (H + G) + H * 128)
            kv, pairs = kv + G * 256, pairs + H * (128 + 256)
        w += D * H * 128 + 3 * D * c["hidden"] + 2 * D * c["side"]
    return w, head, kv / L, pairs / L, L, c["window"] if "a" not in c["pattern"] else 1 << 30


def work(case):
    """Per token of the loop every weight and the visible cache once (a token depends on the one before); a prompt reads the
    weights once; samples share a step's weights."""
    c = case
    linears, head, kv, pairs, L, window = _parts(c)
    es = {"f32": 4.0, "f16": 2.0, "bf16": 2.0, "fp8": 1.0, "int4": 0.5625}[c["dtype"]]
    hs = 4.0 if c["dtype"] == "f32" else 2.0
    weights, kvb = linears * es + head * hs, kv * L * hs
    nbytes = flops = 0.0
    pos = c["cached"]
    if c["new"]:
        seen = sum(min(window, pos + i + 1) for i in range(c["new"]))
        nbytes += weights + (pos + c["new"]) * kvb + c["vocab"] * 4
        flops += 2.0 * linears * c["new"] + 2.0 * head + 2.0 * pairs * L * seen
        pos += c["new"]
    for _ in range(c["scored"] + c["steps"]):
        pos += 1
        nbytes += weights + min(window, pos) * kvb
        flops += c["samples"] * (2.0 * (linears + head) + 2.0 * pairs * L * min(window, pos))
    nbytes += c["scored"] * c["vocab"] * 4
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp32 models differ by the order of their sums; 16-bit caches round keys and values that differ by such sums to other
    # neighbours now and then, and a prompt's 16-bit operand pairs carry about 16 bits; the configured decoders' norms
    # behind every sublayer amplify both
    if case["family"] == "dafidra":
        return {"rel": 2e-2, "max": 1.5e-1, "differ": 0.0}
    if case["family"] == "kazodra":
        return {"rel": 5e-3, "max": 5e-2, "differ": 0.0}
    if case["dtype"] == "f32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.0}
    return {"rel": 2e-3, "max": 2e-2, "differ": 0.0}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
M64 = (1 << 64) - 1
GOLDEN, MUL1, MUL2 = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB


def _signed(v):
    v &= M64
    return v - (1 << 64) if v >> 63 else v


def _mix(z):
    z ^= z >> 30
    z = z * MUL1 & M64
    z ^= z >> 27
    z = z * MUL2 & M64
    return z ^ z >> 31


def _fields(base, k):
    """The sum of the four 16-bit fields of the mixed counter base + k * GOLDEN (int64 tensors, wrapping)."""
    z = base + _signed(k * GOLDEN)
    z ^= (z >> 30) & ((1 << 34) - 1)
    z *= _signed(MUL1)
    z ^= (z >> 27) & ((1 << 37) - 1)
    z *= _signed(MUL2)
    z ^= (z >> 31) & ((1 << 33) - 1)
    s = z & 0xFFFF
    for shift in (16, 32, 48):
        s += (z >> shift) & 0xFFFF
    return s


def synth(seed, uid, rows, cols, std):
    """A seeded matrix as the framework defines it, in fp32: three counter outputs per element, their twelve 16-bit fields
    summed, centred and scaled."""
    key = _mix(seed ^ _mix(uid + GOLDEN & M64))
    out = torch.empty(rows * cols, dtype=torch.float32, device="cuda")
    scale = float(np.float32(std) / np.float32(65536.0))
    for a in range(0, rows * cols, 1 << 25):
        b = min(rows * cols, a + (1 << 25))
        base = torch.arange(a, b, dtype=torch.int64, device="cuda") * _signed(3 * GOLDEN) + _signed(key)
        s = _fields(base, 1) + _fields(base, 2) + _fields(base, 3) - 393210
        out[a:b] = s.to(torch.float32) * scale
    return out.view(rows, cols)


def rounded(w, dtype):
    return (w if dtype == "f32" else w.to(torch.float16) if dtype == "f16" else w.to(torch.bfloat16)).double()


def linear(seed, uid, rows, cols, std, dtype, transpose):
    """A linear's matrix [in, out] in 64 bits as the model holds it; `transpose`: the seeded layout is [out, in]."""
    w = synth(seed, uid, rows, cols, std)
    if dtype not in ("fp8", "int4"):
        return rounded(w, dtype).t() if transpose else rounded(w, dtype)
    w = w if transpose else w.t().contiguous()  # [out, in]
    if dtype == "fp8":
        scale = w.abs().amax(1, keepdim=True) / 448.0
        q = (w / scale).to(torch.float8_e4m3fn)
        return (q.double() * scale.double()).t()
    g = w.view(w.shape[0], -1, 32)
    scale = (g.abs().amax(2, keepdim=True) / 7.0).to(torch.float16).float()
    q = torch.round(g / scale).clamp(-8, 7)
    return (q.double() * scale.double()).view(w.shape).t()


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def attend(q, k, v, scale, window=None, bias=None, sink=None):
    """Causal softmax attention of all positions, [heads, T, d] each (64 bits), a few heads at a time."""
    H, T = q.shape[0], q.shape[1]
    out = torch.empty(H, T, v.shape[2], dtype=torch.float64, device="cuda")
    t = torch.arange(T, device="cuda")
    dist = t[:, None] - t[None, :]
    hidden = (dist < 0) | (dist >= (window or T))
    step = max(1, (1 << 27) // (T * T))
    for a in range(0, H, step):
        s = torch.matmul(q[a:a + step], k[a:a + step].transpose(1, 2)) * scale
        if bias is not None:
            s -= bias[a:a + step, None, None] * dist
        s.masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[a:a + step, None, None].expand(-1, T, 1)], 2)
        p = torch.softmax(s, 2)[:, :, :T]
        out[a:a + step] = torch.matmul(p, v[a:a + step])
    return out


def heads_of(x, heads):
    return x.view(x.shape[0], heads, -1).transpose(0, 1)


def rope32(x, n):
    """Neighbouring pairs of the last axis rotated, the angles of the model's fp32 table; x [heads, T, n]."""
    T = x.shape[1]
    theta = np.arange(T, dtype=np.float32)[:, None] / np.power(np.float32(10000.0), np.float32(2.0) * np.arange(n // 2, dtype=np.float32) / np.float32(n))
    return turn(x, torch.from_numpy(np.cos(theta)).double().cuda(), torch.from_numpy(np.sin(theta)).double().cuda())


def turn(x, cos, sin):
    y = torch.empty_like(x)
    u, v = x[..., 0::2], x[..., 1::2]
    y[..., 0::2], y[..., 1::2] = u * cos - v * sin, v * cos + u * sin
    return y


def silu(x):
    return x * torch.sigmoid(x)


def forward_dense(c, seed, ids):
    D, H, G, hd, L, dt, std = c["dim"], c["heads"], c["kv_heads"], c["hd"], c["layers"], c["dtype"], std_of(c)
    edt = "bf16" if dt in ("fp8", "int4") else dt
    embed = rounded(synth(seed, 0, c["vocab"], D, std), edt)
    x, alpha = embed[ids], 1.0 / math.sqrt(2.0 * L)
    for l in range(L):
        w = lambda which, rows, cols, tr=False: linear(seed, 16 + 16 * l + which, rows, cols, std, dt, tr)  # noqa: E731
        n = rms(x, 1e-5)
        q = rope32(heads_of(n @ w(0, D, H * hd), H), hd)
        k = rope32(heads_of(n @ w(1, D, G * hd), G), hd).repeat_interleave(H // G, 0)
        v = heads_of(n @ w(2, D, G * hd), G).repeat_interleave(H // G, 0)
        o = attend(q, k, v, 1.0 / math.sqrt(hd)).transpose(0, 1).reshape(len(ids), -1)
        x = x + alpha * (o @ w(3, H * hd, D))
        n = rms(x, 1e-5)
        g = n @ w(4, D, c["hidden"])
        g = torch.maximum(g, 0.5 * g) ** 2 if c["activation"] == 1 else silu(g)
        x = x + alpha * ((g * (n @ w(5, D, c["hidden"]))) @ w(6, D, c["hidden"], True))
    return rms(x, 1e-5), embed


def forward_moe(c, seed, ids):
    D, H, L, std, C, Rd, N, V = c["dim"], c["heads"], c["layers"], std_of(c), c["latent"], c["rope"], c["nope"], c["vdim"]
    embed = rounded(synth(seed, 0, c["vocab"], D, std), "bf16")
    x, alpha, T = embed[ids], 1.0 / math.sqrt(2.0 * L), len(ids)
    for l in range(L):
        w = lambda which, rows, cols: rounded(synth(seed, 0x100000 + 1024 * l + which, rows, cols, std), "bf16")  # noqa: E731
        n = rms(x, 1e-5)
        q = heads_of(n @ w(0, D, H * (N + Rd)), H)
        lat = rms(n @ w(1, D, C), 1e-5)
        kr = rope32((n @ w(2, D, Rd))[None], Rd).expand(H, T, Rd)
        k = torch.cat([heads_of(lat @ w(3, C, H * N), H), kr], 2)
        q = torch.cat([q[..., :N], rope32(q[..., N:].contiguous(), Rd)], 2)
        o = attend(q, k, heads_of(lat @ w(4, C, H * V), H), 1.0 / math.sqrt(N + Rd)).transpose(0, 1).reshape(T, -1)
        x = x + alpha * (o @ w(5, H * V, D))
        n = rms(x, 1e-5)
        p = torch.softmax(n @ w(6, D, c["experts"]), 1)
        top = torch.topk(p, c["top"], 1)
        SH = c["shared"] * c["hidden"]
        y = (silu(n @ w(7, D, SH)) * (n @ w(8, D, SH))) @ w(9, D, SH).t()
        for e in range(c["experts"]):
            row, slot = (top.indices == e).nonzero(as_tuple=True)
            if len(row):
                h = n[row]
                f = (silu(h @ w(16 + 3 * e, D, c["hidden"])) * (h @ w(17 + 3 * e, D, c["hidden"]))) @ w(18 + 3 * e, D, c["hidden"]).t()
                y[row] += top.values[row, slot][:, None] * f
        x = x + alpha * y
    return rms(x, 1e-5), embed


def named(seed, std):
    def w(name, out, inp):  # [out, in], keyed by the tensor's name (FNV-1a)
        h = 1469598103934665603
        for ch in name.encode():
            h = (h ^ ch) * 1099511628211 & M64
        return rounded(synth(seed, h, out, inp, std), "bf16")
    return w


def forward_dafidra(c, seed, ids):
    w, D, H, G, T, eps = named(seed, std_of(c)), c["dim"], c["heads"], c["kv_heads"], len(ids), 1e-5
    M = H // 2
    x = w("embed", c["vocab"], D)[ids]
    pos = torch.arange(T, dtype=torch.float64, device="cuda")
    slopes = 2.0 ** (-8.0 * (torch.arange(H, dtype=torch.float64, device="cuda") + 1) / H)
    t = torch.arange(T, device="cuda")
    future = t[None, :] > t[:, None]
    for l in range(c["layers"]):
        p = "l%d.mix.left." % l
        temp = 1.0 + 0.1 * torch.log(torch.floor((pos + 1.0) / 4096.0) + 1.0)
        q = heads_of(rms(x @ w(p + "q", H * 128, D).t(), eps) * temp[:, None], H)
        k = heads_of(rms(x @ w(p + "k", G * 128, D).t(), eps), G).repeat_interleave(H // G, 0)
        v = heads_of(x @ w(p + "v", G * 128, D).t(), G).repeat_interleave(H // G, 0)
        o = attend(q, k, v, 128 ** -0.5, c["window"], slopes, torch.zeros(H, dtype=torch.float64, device="cuda")).transpose(0, 1)
        o = o * torch.sigmoid(x @ w(p + "g", H, D).t())[:, :, None]
        a = rms(o.reshape(T, -1) @ w(p + "o", D, H * 128).t(), eps)
        p = "l%d.mix.right." % l
        q = heads_of(x @ w(p + "q", M * 128, D).t(), M) * 128 ** -0.5
        k = heads_of(x @ w(p + "k", M * 128, D).t(), M)
        v = heads_of(x @ w(p + "v", M * 256, D).t(), M)
        gi = 15.0 * torch.tanh((x @ w(p + "i", M, D).t()) / 15.0)
        gf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w(p + "f", M, D).t() + 3.0) / 15.0))
        F = torch.cumsum(gf, 0).t()  # [M, T]
        out = torch.empty(M, T, 256, dtype=torch.float64, device="cuda")
        for h in range(M):
            d = F[h][:, None] - F[h][None, :] + gi[:, h][None, :]  # log weight of position s at t
            d.masked_fill_(future, -math.inf)
            m = torch.maximum(d.amax(1), F[h])  # the running maximum starts at zero
            s = (q[h] @ k[h].t()) * torch.exp(d - m[:, None])
            out[h] = (s @ v[h]) / (torch.maximum(s.sum(1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        out = rms(out, eps).transpose(0, 1).reshape(T, -1) * torch.sigmoid(x @ w(p + "g", M * 256, D).t())
        b = rms(out @ w(p + "o", D, M * 256).t(), eps)
        x = x + 0.5 * rms((a + b) * 0.5, eps)
        p = "l%d.mlp." % l
        f = (silu(x @ w(p + "gate", c["hidden"], D).t()) * (x @ w(p + "up", c["hidden"], D).t())) @ w(p + "down", D, c["hidden"]).t()
        x = x + 0.5 * rms(f, eps)
    return rms(x, eps), w("head", c["vocab"], D)


def layer_norm(x, eps):
    return rms(x - x.mean(-1, keepdim=True), eps)


def spin(x, rot):
    f = rot["base"] ** (-2.0 * np.arange(rot["dims"] // 2) / rot["dims"])
    s = rot.get("scaling")
    if s:
        n = s["original"] * f / (2.0 * np.pi)
        t = (n - s["low"]) / (s["high"] - s["low"])
        f = np.where(n > s["high"], f, np.where(n < s["low"], f / s["factor"], (1.0 - t) * f / s["factor"] + t * f))
    a = torch.from_numpy(np.arange(x.shape[1])[:, None] * f).cuda()
    return turn(x, torch.cos(a), torch.sin(a))


def forward_kazodra(c, seed, ids):
    w, D, T, eps, cfg = named(seed, std_of(c)), c["dim"], len(ids), 1e-5, kazodra_json(c)
    embed = w("embed", c["vocab"], D)
    x = embed[ids]
    side = w("side.embed", c["vocab"], c["layers"] * c["side"])[ids] if c["side"] else None
    t = torch.arange(T, device="cuda")
    ago = (t[:, None] - t[None, :]).double()
    for l, L in enumerate(cfg["layers"]):
        p, m, H, h = "l%d.mix." % l, L["mixer"], L["mixer"]["heads"], layer_norm(x, eps)
        if L["type"] == "latent_attention":
            q = heads_of(h @ w(p + "q", H * 192, D).t(), H)
            low = h @ w(p + "dkv", 576, D).t()
            lat, kr = rms(low[:, :512], eps), spin(low[:, 512:].contiguous()[None], m["rot"]).expand(H, T, 64)
            q = torch.cat([q[..., :128], spin(q[..., 128:].contiguous(), m["rot"])], 2)
            k = torch.cat([heads_of(lat @ w(p + "uk", H * 128, 512).t(), H), kr], 2)
            o = attend(q, k, heads_of(lat @ w(p + "uv", H * 128, 512).t(), H), m["scale"], c["window"])
            o = o.transpose(0, 1).reshape(T, -1)
        elif L["type"] == "lightning":
            q, k, v = (heads_of(silu(h @ w(p + n, H * 128, D).t()), H) for n in "qkv")
            o = torch.empty(H, T, 128, dtype=torch.float64, device="cuda")
            for a in range(H):
                decay = torch.where(ago >= 0, float(np.float32(m["decay"][a])) ** ago.clamp(min=0), 0.0)
                o[a] = ((q[a] @ k[a].t()) * decay) @ v[a]
            o = rms(o.transpose(0, 1).reshape(T, -1), eps) * torch.sigmoid(h @ w(p + "g", H * 128, D).t())
        else:
            G = m["kv_heads"]
            q = spin(heads_of(h @ w(p + "q", H * 128, D).t(), 2 * H).contiguous(), m["rot"]).view(H, 2, T, 64)
            k = spin(heads_of(h @ w(p + "k", G * 128, D).t(), 2 * G).contiguous(), m["rot"]).view(G, 2, T, 64).repeat_interleave(H // G, 0)
            v = heads_of(h @ w(p + "v", G * 128, D).t(), G).repeat_interleave(H // G, 0)
            o = attend(q[:, 0], k[:, 0], v, m["scale"]) - m["diff"] * attend(q[:, 1], k[:, 1], v, m["scale"])
            o = (rms(o, eps) * (1.0 - m["diff"])).transpose(0, 1).reshape(T, -1) * torch.sigmoid(h @ w(p + "g", H * 128, D).t())
        x = x + layer_norm(o @ w(p + "o", D, H * 128).t(), eps)
        p, h = "l%d.mlp." % l, layer_norm(x, eps)
        x = x + layer_norm((silu(h @ w(p + "gate", c["hidden"], D).t()) * (h @ w(p + "up", c["hidden"], D).t())) @ w(p + "down", D, c["hidden"]).t(), eps)
        if c["side"]:
            p, z = "l%d.side." % l, x @ w("l%d.side.gate" % l, c["side"], D).t()
            g = torch.nn.functional.gelu(z, approximate="tanh") * side[:, l * c["side"]:(l + 1) * c["side"]]
            x = x + rms(g @ w(p + "proj", D, c["side"]).t(), eps)
    return layer_norm(x, eps), embed


FORWARD = {"dense": forward_dense, "moe": forward_moe, "dafidra": forward_dafidra, "kazodra": forward_kazodra}


def exact(case, seed):
    """The logits of run() in 64 bits, on the weights as stored (rounded, quantised) and an unrounded cache; ids have none."""
    c = case
    (cached, new, scored, _), _ = tokens_of(c, seed)
    ids = np.concatenate([cached, new, scored]).astype(np.int64)
    with torch.no_grad():
        hidden, head = FORWARD[c["family"]](c, seed + 1, torch.from_numpy(ids).cuda())
        at = c["cached"] + c["new"]
        wanted = [at - 1] * (c["new"] > 0) + list(range(at, at + c["scored"]))
        logits = (hidden[wanted] @ head.t()).cpu().numpy()
    out = {}
    if c["new"]:
        out["prompt_logits"], logits = logits[0], logits[1:]
    if c["scored"]:
        out["scored_logits"] = list(logits)
    if c["steps"]:
        out["ids"] = None
    return out
