"""The steps whose speed is watched: what the engine does for serving and for replaying traces.

A case is one batch: requests that decode one token each, prompts or portions of prompts, or both in one step. A decode step runs as the
engine runs it, replayed from the graphs of ``DecodeGraphs``, with the one synchronisation that brings its tokens to the host; every other
step goes through ``ModelRunner.step``, which generation and trace replay both drive. Models have random weights at the two layer sizes that
``bench.py`` compares designs at (2,048 and 4,096 wide, eight layers; 4,096 wide are the layers of the 8B Qwen3 model, and a vocabulary of
32,768 keeps the head's share of a step as it is in the 36-layer model). Five designs: the dense Qwen3 decoder, and the four that hold most
other kinds of token mixing between them: Radapel (Mamba-2, chunks with a distance bias, latent attention), Verorax (delta rule, differential
and latent attention, token shift), Finolix (several residual streams, windowed latent attention, gated attention, routed experts) and Nidudra
(gated linear attention, windows with kept first keys, sinks). Routed experts are Finolix's alone here: with random weights a token's last
chosen expert is often a near-tie, and in the designs that norm every sublayer's output one other choice moves that token's logits by far more
than rounding does, so that nothing could be compared.

Fields of a case: ``model``, ``width``, ``dtype``; ``decode`` requests with contexts of up to ``context`` tokens (all alike, or spread evenly
from an eighth of it where ``uneven``); ``prompts`` prompts that bring ``tokens`` tokens in all, each with ``cached`` tokens of its own in the
cache already; ``every``: logits are wanted for each decoded token, and along a prompt for every so-manieth token and the last.
"""

import hashlib
import math
import random

import torch
import torch.nn.functional as F

from oxr_inference_b200 import ops
from oxr_inference_b200.engine.batch import StepEntry
from oxr_inference_b200.engine.graphs import DecodeGraphs
from oxr_inference_b200.engine.runtime import ModelRunner
from oxr_inference_b200.weights.random_init import shape_only_model

LAYERS, VOCAB, PAGE, HEAD = 8, 32768, 16, 128
MODELS = ("qwen3", "radapel", "verorax", "finolix", "nidudra")


def case(name, model, width, *, dtype="bfloat16", decode=0, context=0, uneven=False, prompts=0, tokens=0, cached=0, every=32):
    out = {} if name is None else {"name": name}
    out.update(model=model, width=width, dtype=dtype, decode=decode, context=context, uneven=uneven, prompts=prompts, tokens=tokens, cached=cached, every=every)
    return out


def listed():
    return [
        # one user alone with a small model: a short chat, where the length of the chain of launches counts
        case("qwen3_decode_1", "qwen3", 2048, decode=1, context=200),
        # the benchmark's decode step: eight requests with 2,048 tokens of context each
        case("qwen3_decode_8", "qwen3", 4096, decode=8, context=2048),
        # a busy server: requests of very different lengths, a batch that fills no power of two
        case("qwen3_decode_uneven", "qwen3", 4096, decode=48, context=4000, uneven=True),
        # the benchmark's prompt: 2,048 tokens in one step
        case("qwen3_prompt", "qwen3", 4096, prompts=1, tokens=2048),
        # continuous batching: a ragged portion of a long prompt beside requests that decode
        case("qwen3_mixed", "qwen3", 4096, decode=31, context=1500, uneven=True, prompts=1, tokens=1531, cached=517),
        # a trace replayed in true 32 bits, to compare logits
        case("qwen3_replay_fp32", "qwen3", 2048, dtype="float32", prompts=1, tokens=333, every=8),
        # the other designs: a prompt of the benchmark's length, ragged prompts together, decoding, portions beside decoding
        case("radapel_prompt", "radapel", 4096, prompts=1, tokens=2048),
        case("radapel_decode_8", "radapel", 4096, decode=8, context=2048),
        case("verorax_prompts", "verorax", 4096, prompts=3, tokens=2011),
        case("verorax_decode_uneven", "verorax", 4096, decode=13, context=1800, uneven=True),
        case("finolix_mixed", "finolix", 4096, decode=20, context=1700, uneven=True, prompts=2, tokens=1401, cached=300),
        case("nidudra_prompt", "nidudra", 4096, prompts=1, tokens=2048),
    ]


def spread(rng, low, high):
    """A whole number whose logarithm is uniform."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    model, width = rng.choice(MODELS), rng.choice((2048, 4096))
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "mixed"))
    if model == "qwen3" and kind == "prompt" and rng.random() < 0.3:
        return case(None, model, 2048, dtype="float32", prompts=rng.randint(1, 2), tokens=spread(rng, 40, 333), every=8)
    out = case(None, model, width, every=rng.choice((16, 32, 64)))
    if kind != "prompt":
        out.update(decode=spread(rng, 1, 48 if kind == "decode" else 24), context=spread(rng, 100, 2200), uneven=rng.random() < 0.6)
    if kind != "decode":
        out.update(prompts=rng.randint(1, 4), tokens=spread(rng, 150, 1900), cached=rng.choice((0, 0, spread(rng, 16, 600))))
    return out


# ------------------------------------------------------------------------------------------------ models
def config(model, width):
    """The designs at one size, as ``bench.py`` sets them beside each other."""
    heads, kv, ff = width // HEAD, width // HEAD // 4, {2048: 8192, 4096: 12288}[width]
    sizes = {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5}
    dense = {"kind": "dense", "ff": ff}
    if model == "qwen3":
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_size": width, "intermediate_size": ff,
                "num_hidden_layers": LAYERS, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": HEAD, "rms_norm_eps": 1e-6,
                "rope_theta": 1000000.0, "vocab_size": VOCAB, "tie_word_embeddings": False, "max_position_embeddings": 8192}
    base = {"norm": {"eps": 1e-6}, "vocab": VOCAB, "width": width}
    latent = {"heads": heads, "dim": HEAD, "rot_dim": 64, "rot": {"dims": 64, "base": 10000.0}, "vdim": HEAD, "kv_rank": 192, "scale": (HEAD + 64) ** -0.5}
    if model == "radapel":
        mlp = {**dense, "limit": 7.0}
        chunked = {**sizes, "mask": {"size": 1024}, "bias_max": 512, "bias_rows": 32}
        mamba = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
        turn = (("mamba2", mamba, mlp), ("attention", chunked, mlp), ("attention", chunked, mlp), ("latent_attention", latent, mlp))
        base.update(architecture="Radapel", embedding={"scale": 1.0})
    elif model == "verorax":
        latent["q_rank"] = width // 4
        diff = {**sizes, "dim": HEAD // 2, "diff": 0.4, "scale": (HEAD // 2) ** -0.5, "mask": {"size": 1024}}
        pair = {"left": {**sizes, "mask": {"size": 1024}, "rot": {"dims": HEAD // 2, "base": 100000.0}},
                "right": {"heads": width // 128, "dim": 128, "rank": 64}, "left_scale": 0.7, "right_scale": 0.6}
        turn = (("latent_attention", latent, dense), ("attention", diff, dense), ("parallel", pair, dense), ("latent_attention", latent, dense))
        base.update(architecture="Verorax")
    elif model == "finolix":
        latent["q_rank"], latent["mask"] = width // 4, {"size": 1024}
        latent["rot"] = {"dims": 64, "base": 10000.0, "scaling": {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        gated = {**sizes, "rot": {"dims": HEAD // 4, "base": 100000.0}}
        mlps = ({"kind": "dense", "ff": ff * 3 // 2}, {"kind": "moe", "expert": {"ff": ff // 8}, "router": {"experts": 16, "top": 4}})
        turn = tuple((k, m, mlp) for mlp in mlps for k, m in (("latent_attention", latent), ("attention", gated)))
        base.update(architecture="Finolix", streams=2)
    else:
        windowed = {**sizes, "mask": {"size": 1024, "keep_first": 64}}
        sinked = {**sizes, "rot": {"dims": HEAD // 2, "base": 100000.0, "scaling": {"factor": 4.0, "low": 1.0, "high": 8.0, "original": 2048}}}
        pair = {"left": {**sizes, "conv": 4, "rot": {"dims": HEAD // 2, "base": 10000.0, "scaling": {"factor": 4.0, "original": 1024, "fast": 16.0, "slow": 2.0}}},
                "right": {"heads": width // 256, "dim": 128, "vdim": 256, "tau": 8.0, "rank": 64}}
        turn = (("attention", windowed, dense), ("attention_2", sinked, dense), ("parallel", pair, dense), ("attention", windowed, dense))
        base.update(architecture="Nidudra", logit_softcap=50.0)
    layers = []
    for i in range(LAYERS):
        kind, mixer, mlp = turn[i % 4]
        if model == "nidudra" and i % 4 == 3:
            mixer = {**mixer, "kv_from": i - 3}
        layers.append({"type": kind, "mixer": mixer, "mlp": mlp})
    return {**base, "layers": layers}


def lengths(case):
    """[(tokens in the cache, tokens of this step)] of every request: the decoding ones, then the prompts."""
    n, top = case["decode"], case["context"]
    low = top // 8 if case["uneven"] and n > 1 else top
    out = [(max(1, low + round(i * (top - low) / max(n - 1, 1))), 1) for i in range(n)]
    left, p = case["tokens"], case["prompts"]
    for i in range(p):   # shares of 3 : 5 : 7 : 9, the last takes the rest
        n = left if i == p - 1 else max(1, case["tokens"] * (3 + 2 * i) // sum(3 + 2 * j for j in range(p)))
        left -= n
        out.append((case["cached"], n))
    return out


def wanted(case, tokens):
    return sorted({*range(case["every"] - 1, tokens, case["every"]), tokens - 1})


def sequences(case, seed):
    rng = random.Random(seed)
    return [[rng.randrange(VOCAB) for _ in range(a + b)] for a, b in lengths(case)]


def prepare(case, seed):
    """A loaded model, the requests with their contexts in the cache, and for decode steps the graphs that a server keeps."""
    sizes, ids = lengths(case), sequences(case, seed)
    pages = 8 + sum((a + b) // PAGE + 2 for a, b in sizes)
    runner = ModelRunner.from_config(config(case["model"], case["width"]), seed, dtype=case["dtype"], page_size=PAGE, num_pages=pages, max_requests=len(sizes),
                                     max_positions=8192)
    cache, entries, fresh = runner.cache, [], []
    for i, ((before, now), seq) in enumerate(zip(sizes, ids)):
        if before == 0:
            fresh.append((i, seq, wanted(case, now)))
            continue
        request = cache.open(f"r{i}")
        assert cache.reserve(request, before + now)
        for at in range(0, before, 2048):
            runner.step([StepEntry(request, seq[at:min(at + 2048, before)], [])])
        entries.append(StepEntry(request, seq[before:], wanted(case, now)))
    runner.check()
    graphs = None if case["prompts"] else Graphs(runner, max_batch=len(entries), max_positions=8192)
    return {"runner": runner, "entries": entries, "fresh": fresh, "graphs": graphs}


class Graphs(DecodeGraphs):
    """The graphs of decode steps, with the logits that the tokens are chosen from in reach."""

    def _forward(self, ctx):
        self.logits = self.runner.model.step(ctx, self.runner.cache)
        s = ctx.sampling
        return ops.sample(self.logits, s["temperature"], s["seed_lo"], s["seed_hi"], s["counter"])


def run(state):
    """One step. Prompts with nothing cached come and go with it; the other requests stay where they are (a recurrent state moves on)."""
    runner, entries = state["runner"], list(state["entries"])
    if state["graphs"] is not None:
        state["graphs"].run(entries)
        torch.cuda.current_stream().synchronize()   # the chosen tokens are on the host now; near-ties, so it is their logits that come back
        return state["graphs"].logits[:len(entries)]
    opened = []
    for i, seq, want in state["fresh"]:
        request = runner.cache.open(f"r{i}")
        assert runner.cache.reserve(request, len(seq))
        opened.append(request)
        entries.append(StepEntry(request, seq, want))
    logits = runner.step(entries, advance=False)
    for request in opened:
        runner.cache.close(request)
    return logits


# ------------------------------------------------------------------------------------------------ what a step cannot do without
def work(case):
    c = config(case["model"], case["width"])
    sizes = lengths(case)
    new, rows = sum(b for _, b in sizes), sum(len(wanted(case, b)) for _, b in sizes)
    size = 4 if case["dtype"] == "float32" else 2
    weights = products = 0
    for name, (_, _, info) in shape_only_model(c).named_parameters().items():
        n = math.prod(info.shape)
        if name.startswith(("embed", "model.embed")):
            weights += new * case["width"]
        elif ".mlp.e" in name:      # 4 experts of 16 for each token
            weights += n * (1 - (3 / 4) ** new)
            products += n / 4 * new
        else:
            weights += n
            products += n * (rows if "head" in name else new)
    kinds = [("full", None)] * LAYERS if case["model"] == "qwen3" else [(layer["type"], layer["mixer"]) for layer in c["layers"]]
    heads, kv = case["width"] // HEAD, case["width"] // HEAD // 4
    keys = [sum(range(a + 1, a + b + 1)) for a, b in sizes]                         # (query, key) pairs of a causal layer
    near = [sum(min(j, 1024) for j in range(a + 1, a + b + 1)) for a, b in sizes]   # the same with the last 1,024 keys only
    moved = flops = 0
    for kind, mixer in kinds:
        limit = bool(mixer) and "mask" in mixer.get("left", mixer)
        pairs = sum(near if limit else keys)
        read = sum((min(a + b, 1024 + b) if limit else a + b) for a, b in sizes)
        if kind == "latent_attention":
            flops += 2 * pairs * heads * (2 * HEAD + 64)
            moved += (read + new) * 256
        elif kind != "mamba2":
            flops += 4 * pairs * heads * HEAD * (1.5 if mixer and "diff" in mixer else 1)
            moved += (read + new) * 2 * kv * HEAD
        state = {"mamba2": 2 * case["width"] * 128, "parallel": case["width"] * 128}.get(kind, 0)
        flops += 6 * new * state
        moved += 2 * len(sizes) * state * (4 // size)
    return {"bytes": weights * size + moved * size + rows * VOCAB * 4, "flops": 2 * products + flops}


def tolerance(case):
    """Errors against 64 bits were 7e-6 for the 32-bit model, 0.02 for Qwen3, 0.005 for Finolix and 0.006 to 0.015 for the others in bfloat16."""
    if case["dtype"] == "float32":
        return {"rel": 3e-5}
    return {"rel": 0.02 if case["model"] == "finolix" else 0.03}


# ------------------------------------------------------------------------------------------------ the same logits in 64 bits
class Weights:
    """Random weights as they are drawn for a loaded model: by seed and name, on the device, stored in bfloat16."""

    def __init__(self, seed):
        self.seed = seed

    def __call__(self, name, *shape, one=False):
        digest = hashlib.sha256(f"{self.seed}:{name}".encode()).digest()
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int.from_bytes(digest[:8], "little") & 0x7FFF_FFFF_FFFF_FFFF)
        t = torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda")
        return (1.0 + 0.1 * t if one else 0.02 * t).to(torch.bfloat16).double()


class Part:
    """The tensors under one prefix; ``p(x, name, rows)`` is the product with a matrix."""

    def __init__(self, w, prefix):
        self.w, self.prefix = w, prefix

    def sub(self, prefix):
        return Part(self.w, self.prefix + prefix)

    def vec(self, name, *shape):
        return self.w(self.prefix + name, *shape)

    def norm(self, name, n):
        return self.w(self.prefix + name, n, one=True)

    def __call__(self, x, name, rows):
        return x @ self.w(self.prefix + name, rows, x.shape[-1]).T


def rms(x, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def heads_of(x, n):
    return x.reshape(x.shape[0], n, -1)


def frequencies(dims, base, scaling=None):
    """One frequency per pair and the factor on cos and sin: plain, slowed in three bands of wavelength, or along a ramp over the pairs."""
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not scaling:
        return f, 1.0
    factor, original = scaling["factor"], scaling["original"]
    if "low" in scaling:
        def blend(x):
            t = (original * x / (2 * math.pi) - scaling["low"]) / (scaling["high"] - scaling["low"])
            return min(max(t, 0.0), 1.0)
        return [x * (blend(x) + (1 - blend(x)) / factor) for x in f], 1.0
    at = [dims * math.log(original / (2 * math.pi * scaling[k])) / (2 * math.log(base)) for k in ("fast", "slow")]
    low, high = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    ramp = [min(max((i - low) / max(high - low, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [x * (r / factor + 1 - r) for x, r in zip(f, ramp)], 0.1 * math.log(factor) + 1.0


def rotate(x, rot, neighbours=False, single=False):
    """[T, heads, D]: the first pairs of each head turn with the position (``single``: the angles are made in 32 bits, as the Qwen3 model defines them)."""
    freq, stretch = frequencies(rot["dims"], rot["base"], rot.get("scaling"))
    n, kind = len(freq), torch.float32 if single else torch.float64
    if single:
        f = 1.0 / (rot["base"] ** (torch.arange(0, 2 * n, 2, dtype=torch.float) / (2 * n)))
    else:
        f = torch.tensor(freq, dtype=kind)
    angle = torch.outer(torch.arange(x.shape[0], dtype=kind), f)
    cos, sin = ((t(angle) * stretch).double().cuda()[:, None, :] for t in (torch.cos, torch.sin))
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if neighbours else (x[..., :n], x[..., n:2 * n])
    a, b = u * cos - v * sin, v * cos + u * sin
    turned = torch.stack((a, b), -1).flatten(-2) if neighbours else torch.cat((a, b), -1)
    return torch.cat((turned, x[..., 2 * n:]), -1)


def attend(q, k, v, scale, *, window=0, keep_first=0, chunk=0, sink=None, bias=None):
    """q [T, H, D], k [T, G, D], v [T, G, DV] -> [T, H, DV], a group of heads at a time. ``bias``: [distances, H]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device="cuda")
    back = i[:, None] - i[None, :]
    seen = back >= 0
    if window:
        seen &= (back < window) | (i < keep_first)[None, :]
    if chunk:
        seen &= (i // chunk)[:, None] == (i // chunk)[None, :]
    out, step = [], H // G
    for h in range(0, H, step):
        kk, vv = k[:, h // step], v[:, h // step]
        s = torch.einsum("thd,sd->hts", q[:, h:h + step], kk) * scale
        if bias is not None:
            s += bias[:, h:h + step].T[:, back.clamp(0, bias.shape[0] - 1)]
        s.masked_fill_(~seen, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[h:h + step, None, None].expand(-1, T, 1)), -1)
        s = torch.softmax(s, -1)[..., :T]
        out.append(torch.einsum("hts,sd->thd", s, vv))
    return torch.cat(out, 1)


def latent_attention(h, p, m, neighbours, sink):
    """Keys and values are maps of one normed row a token, the rotated part of the keys is shared by the heads."""
    T, H, D, R, L = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    latent = rms(p(h, "dq", m["q_rank"])) * p.norm("dq.norm", m["q_rank"]) if "q_rank" in m else h
    q = heads_of(p(latent, "uq" if "q_rank" in m else "q", H * (D + R)), H)
    down = p(h, "dkv", L + R)
    c = rms(down[:, :L]) * p.norm("dkv.norm", L)
    q = torch.cat((q[..., :D], rotate(q[..., D:], m["rot"], neighbours)), -1)
    k = torch.cat((heads_of(p(c, "uk", H * D), H), rotate(down[:, None, L:], m["rot"], neighbours).expand(T, H, R)), -1)
    v = heads_of(p(c, "uv", H * m["vdim"]), H)
    o = attend(q, k, v, m["scale"], window=m.get("mask", {}).get("size", 0), sink=p.vec("sink", H) if sink else None)
    return p(o.reshape(T, -1), "o", h.shape[1])


def mamba2(h, p, m):
    T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner, wide = H * P, H * P + 2 * G * N
    z, xbc, dt = p(h, "in", inner + wide + H).split((inner, wide, H), -1)
    conv = F.conv1d(F.pad(xbc.T[None], (m["conv"] - 1, 0)), p.vec("conv", wide, m["conv"])[:, None], p.vec("conv.b", wide), groups=wide)[0].T
    x, B, C = F.silu(conv).split((inner, G * N, G * N), -1)
    x, B, C = x.view(T, H, P), *(t.reshape(T, G, 1, N).expand(T, G, H // G, N).reshape(T, H, N) for t in (B, C))
    dt = F.softplus(dt + p.vec("dt_bias", H), threshold=1e9)
    decay = torch.exp(-torch.exp(p.vec("A_log", H)) * dt)
    S, y = torch.zeros(H, N, P, dtype=h.dtype, device="cuda"), torch.empty_like(x)
    fed = dt[..., None] * x
    for t in range(T):
        S = decay[t, :, None, None] * S + B[t, :, :, None] * fed[t, :, None, :]
        y[t] = (C[t, :, None, :] @ S)[:, 0]
    y = (y + p.norm("D", H)[:, None] * x).reshape(T, inner) * F.silu(z)
    return p(rms(heads_of(y, m["norm_groups"])).reshape(T, inner) * p.norm("norm", inner), "o", h.shape[1])


def gated_linear(h, p, m):
    T, H, D, V = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q, k, v = heads_of(p(h, "q", H * D), H) * D ** -0.5, heads_of(p(h, "k", H * D), H), heads_of(p(h, "v", H * V), H)
    alpha = heads_of(torch.sigmoid(p(p(h, "a1", m["rank"]), "a2", H * D) + p.vec("a2.b", H * D)) ** (1.0 / m["tau"]), H)
    S, o = torch.zeros(H, D, V, dtype=h.dtype, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S = alpha[t, :, :, None] * S + k[t, :, :, None] * v[t, :, None, :]
        o[t] = (q[t, :, None, :] @ S)[:, 0]
    o = (rms(o) * p.norm("norm", V)).reshape(T, -1)
    return p(o * F.silu(p(h, "g", H * V)), "o", h.shape[1])


def delta_rule(h, p, m):
    T, H, D = h.shape[0], m["heads"], m["dim"]
    W = H * D
    r, k, v = (heads_of(p(h, n, W), H) for n in ("r", "k", "v"))
    z = p(torch.tanh(p(h, "w1", m["rank"])), "w2", W) + p.vec("w0", W)
    decay = heads_of(torch.exp(-math.exp(-0.5) * torch.sigmoid(z)), H)
    unit = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    out = heads_of(torch.sigmoid(p(h, "a", W) + p.vec("a.b", W)), H) * unit
    S, o = torch.zeros(H, D, D, dtype=h.dtype, device="cuda"), torch.empty_like(v)
    for t in range(T):
        held = unit[t, :, None, :] @ S
        S = decay[t, :, :, None] * S - out[t, :, :, None] * held + k[t, :, :, None] * v[t, :, None, :]
        o[t] = (r[t, :, None, :] @ S)[:, 0]
    o = rms(o).reshape(T, -1) * p.norm("norm", W) * torch.sigmoid(p(h, "g", W))
    return p(o, "o", h.shape[1])


def attention(h, p, m, model, kind, lent):
    """The designs' other softmax attentions. ``lent``: keys and values of the layer that this one reads, and where it leaves its own."""
    T, H, G, D = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    width = h.shape[1]
    if "diff" in m:
        q, k = (heads_of(p(h, n, 2 * c * D) + p.vec(n + ".b", 2 * c * D), 2 * c) for n, c in (("q", H), ("k", G)))
        v = heads_of(p(h, "v", G * m["vdim"]) + p.vec("v.b", G * m["vdim"]), G)
        lq1, lk1, lq2, lk2 = (p.vec(n, D) for n in ("lq1", "lk1", "lq2", "lk2"))
        share = torch.exp((lq1 * lk1).sum()) - torch.exp((lq2 * lk2).sum()) + m["diff"]
        one, two = (attend(q[:, j::2], k[:, j::2], v, m["scale"], window=m["mask"]["size"]) for j in (0, 1))
        return p((rms(one - share * two) * (1.0 - m["diff"])).reshape(T, -1), "o", width)
    q = p(h, "q", H * D)
    if "kv_from" in m:
        q = rms(heads_of(q, H)) * p.norm("q.norm", D)
        k, v = lent["kv"]
    elif "conv" in m:
        k, filtered = p(h, "k", G * D), []
        for name, x in (("q", q), ("k", k)):
            x = x + p.vec(name + ".b", x.shape[1])
            filtered.append(F.conv1d(F.pad(x.T[None], (m["conv"] - 1, 0)), p.vec(name + ".conv", x.shape[1], m["conv"])[:, None], groups=x.shape[1])[0].T)
        q, k, v = heads_of(filtered[0], H), heads_of(filtered[1], G), heads_of(filtered[1], G)
    else:
        q, k, v = heads_of(q, H), heads_of(p(h, "k", G * D), G), heads_of(p(h, "v", G * D), G)
    if kind == "attention_2":
        q, k = (rms(rotate(x, m["rot"])) for x in (q, k))
    elif "kv_from" not in m and model != "radapel":
        q, k = rms(q) * p.norm("q.norm", D), rms(k) * p.norm("k.norm", D)
        if "rot" in m:
            q, k = rotate(q, m["rot"], single=model == "qwen3"), rotate(k, m["rot"], single=model == "qwen3")
    lent["kv"] = k, v
    mask = m.get("mask", {})
    if model == "radapel":
        rows, far = m["bias_rows"], m["bias_max"]
        half = rows // 2
        bucket = [n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(far / half) * (rows - half))) for n in range(far + 1)]
        o = attend(q, k, v, m["scale"], chunk=mask["size"], bias=p.vec("rel", rows, H)[torch.tensor(bucket, device="cuda")])
    else:
        if "left_of_verorax" in m:
            q = q * p.vec("temp", H)[:, None]
        o = attend(q, k, v, m["scale"], window=mask.get("size", 0), keep_first=mask.get("keep_first", 0), sink=p.vec("sink", H) if kind == "attention_2" else None)
        if kind == "attention_2" or model == "finolix" or "left_of_verorax" in m:
            o = o * torch.sigmoid(p(h, "g", H))[:, :, None]
        elif model == "nidudra" and "conv" not in m:
            o = o * torch.sigmoid(heads_of(p(h, "g", H * D), H))
    return p(o.reshape(T, -1), "o", width)


def mix(h, p, layer, model, lent):
    kind, m = layer["type"], layer["mixer"]
    if kind == "mamba2":
        return mamba2(h, p, m)
    if kind == "latent_attention":
        return latent_attention(h, p, m, neighbours=model != "verorax", sink=model != "verorax")
    if kind != "parallel":
        return attention(h, p, m, model, kind, lent)
    if model == "verorax":
        left = attention(h, p.sub("left."), {**m["left"], "left_of_verorax": True}, model, kind, {})
        return m["left_scale"] * left + m["right_scale"] * delta_rule(h, p.sub("right."), m["right"])
    left, right = attention(h, p.sub("left."), m["left"], model, kind, {}), gated_linear(h, p.sub("right."), m["right"])
    return 0.5 * (rms(left) * p.norm("left.out", h.shape[1]) + rms(right) * p.norm("right.out", h.shape[1]))


def unit(h, p, ff, act=F.silu):
    return p(act(p(h, "gate", ff)) * p(h, "up", ff), "down", h.shape[1])


def feed_forward(h, p, mlp, model):
    width = h.shape[1]
    if mlp["kind"] == "dense":
        if model == "radapel":
            gate, up = p(h, "gate", mlp["ff"]).clamp(max=mlp["limit"]), p(h, "up", mlp["ff"]).clamp(-mlp["limit"], mlp["limit"])
            return p(gate * torch.sigmoid(1.702 * gate) * (up + 1), "down", width)
        if model == "finolix":
            return p(F.relu(p(h, "up", mlp["ff"])).square(), "down", width)
        return unit(h, p, mlp["ff"], (lambda z: F.gelu(z, approximate="tanh")) if model == "verorax" else F.silu)
    r = mlp["router"]
    best = torch.topk(p(h, "router", r["experts"]) + p.vec("router.b", r["experts"]), r["top"], -1)
    share, out = torch.softmax(best.values, -1), torch.zeros_like(h)
    for e in range(r["experts"]):
        rows, place = (best.indices == e).nonzero(as_tuple=True)
        if rows.numel():
            out.index_add_(0, rows, share[rows, place][:, None] * unit(h[rows], p.sub(f"e{e}."), mlp["expert"]["ff"]))
    return out


def logits_of(c, model, seed, ids, rows):
    """Logits of ``rows`` of one whole sequence."""
    w = Weights(seed)
    top = Part(w, "")
    if model == "qwen3":
        width, H = c["hidden_size"], c["num_attention_heads"]
        mixer = {"heads": H, "kv_heads": c["num_key_value_heads"], "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "rot": {"dims": HEAD, "base": c["rope_theta"]}}
        x = w("model.embed_tokens.weight", VOCAB, width)[ids]
        for i in range(LAYERS):
            p = Part(w, f"model.layers.{i}.")
            names = {"q": "q_proj.weight", "k": "k_proj.weight", "v": "v_proj.weight", "o": "o_proj.weight", "q.norm": "q_norm.weight", "k.norm": "k_norm.weight",
                     "gate": "gate_proj.weight", "up": "up_proj.weight", "down": "down_proj.weight"}
            at, ff = Named(w, p.prefix + "self_attn.", names), Named(w, p.prefix + "mlp.", names)
            x = x + attention(rms(x) * p.norm("input_layernorm.weight", width), at, mixer, model, "full", {})
            x = x + unit(rms(x) * p.norm("post_attention_layernorm.weight", width), ff, c["intermediate_size"])
        return Part(w, "lm_head.")(rms(x[rows]) * w("model.norm.weight", width, one=True), "weight", VOCAB)
    width = c["width"]
    x = w("embed", VOCAB, width)[ids]
    if model == "finolix":
        x, n = torch.stack([x] * c["streams"]), c["streams"]
    lent = {}
    for i, layer in enumerate(c["layers"]):
        p = Part(w, f"l{i}.")
        own = lent.setdefault(layer["mixer"].get("kv_from", i), {})
        mixer, ff = (lambda h: mix(h, p.sub("mix."), layer, model, own)), (lambda h: feed_forward(h, p.sub("mlp."), layer["mlp"], model))
        for k, part in ((1, mixer), (2, ff)):
            if model == "finolix":
                h = rms((p.vec(f"hc{k}.in", n)[:, None, None] * x).sum(0)) * (1 + p.vec(f"norm{k}", width))
                y = part(h) * p.vec(f"ls{k}", width)
                x = torch.einsum("st,sab->tab", p.vec(f"hc{k}.mix", n, n), x) + p.vec(f"hc{k}.out", n)[:, None, None] * y
            elif model == "nidudra":
                x = x + rms(part(x)) * p.norm(f"norm{k}", width)
            else:
                h = rms(x) * p.norm(f"norm{k}", width)
                if model == "verorax" and k == 1:
                    h = h + (F.pad(h, (0, 0, 1, 0))[:-1] - h) * p.vec("shift", width)
                x = x + rms(part(h)) * p.norm(f"norm{k}b", width)
    x = x.sum(0) if model == "finolix" else x
    last = rms(x[rows]) * ((1 + w("final.norm", width)) if model == "finolix" else w("final.norm", width, one=True))
    out = top(last, "head", VOCAB)
    return 50.0 * torch.tanh(out / 50.0) if model == "nidudra" else out


class Named(Part):
    """A part whose tensors have other names in the checkpoint."""

    def __init__(self, w, prefix, names):
        super().__init__(w, prefix)
        self.names = names

    def norm(self, name, n):
        return super().norm(self.names[name], n)

    def __call__(self, x, name, rows):
        return super().__call__(x, self.names[name], rows)


def exact(case, seed):
    sizes = lengths(case)
    total, longest = sum(a + b for a, b in sizes), max(a + b for a, b in sizes)
    scans = 0 if case["model"] in ("qwen3", "finolix") else 2
    # 64-bit products at about 25 TFLOP/s; a scan is a chain of small launches for each token
    if total * LAYERS * (case["width"] / 4096) ** 2 * 1e9 / 25e12 + scans * total * 1e-4 + len(sizes) * 0.2 > 18 or longest > 8192:
        return None
    c, out = config(case["model"], case["width"]), []
    with torch.inference_mode():
        for (a, b), ids in zip(sorted_requests(sizes), sorted_requests(sequences(case, seed), sizes)):
            rows = [a + i for i in wanted(case, b)]
            out.append(logits_of(c, case["model"], seed, torch.tensor(ids, device="cuda"), rows))
    return torch.cat(out)


def sorted_requests(values, sizes=None):
    """In the order of a step's entries: requests with something cached first."""
    sizes = values if sizes is None else sizes
    return [v for v, s in zip(values, sizes) if s[0]] + [v for v, s in zip(values, sizes) if not s[0]]
