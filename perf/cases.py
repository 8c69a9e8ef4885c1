"""The work that this framework is used for, as cases that can be timed and checked.

A case is a model served by ``Engine`` in one of the three ways in which a program uses it:

  prefill   ``Engine.step`` with whole prompts, the logits of every prompt's last token, the requests ended: how a prompt batch enters, and what a
            replay of given tokens does;
  decode    one captured decode step (``Engine.capture`` and ``replay``, what ``Engine.generate`` runs once per token): packed inputs from pinned memory,
            all layers, sampling, tokens back to pinned memory;
  serve     ``Engine.step`` called as continuous batching calls it: every step carries the next token of each running request and, within a row budget,
            portions of the prompts of the others.

The models are this repository's presets with random weights: the Llama shapes of 1 and 8 G parameters (the headline benchmark is the decode step of the latter
at 8 rows), Nubosun (selective scan, latent attention; bf16 and full fp32) and Bobarax (fixed-decay recurrence, windowed and chunked attention, experts chosen by
token id).  Designs whose experts are chosen by comparing numbers are left out: two correct
implementations differ by whole experts where two router values are close.

What the tokens are does not change what is computed (generated tokens are given, not fed back), so that logits can be compared.
"""
import math
import zlib

import numpy as np
import torch
import torch.nn.functional as F

from libtbvcoll_b200.engine.engine import Engine
from libtbvcoll_b200.models.config import BobaraxConfig, LightningSpec, MambaSpec, ModelConfig, NubosunConfig, TableMoeSpec, get_config
from libtbvcoll_b200.utils.weights import tensor_shapes

DEVICE = "cuda:0"
CHUNK = 4096                 # rows of one pass over a prompt batch, as the benchmark sets them


def _case(model, kind, rows, shortest, longest, dtype="bfloat16", new=0, budget=0):
    return {"model": model, "dtype": dtype, "kind": kind, "rows": rows, "shortest": shortest, "longest": longest, "new": new, "budget": budget}


def listed():
    return [dict(c, name=n) for n, c in {
        # one interactive user of a small model, short context: latency of the launches
        "llama-2k decode 1": _case("llama3-2k", "decode", 1, 100, 100),
        # one user of an 8 G model: weight streaming
        "llama-8b decode 1": _case("llama3-8b", "decode", 1, 512, 512),
        # the headline benchmark's step: eight sequences that were prompts of 512 tokens
        "llama-8b decode 8": _case("llama3-8b", "decode", 8, 512, 512),
        # many users with long, unequal contexts: the cache is several times the weights
        "llama-2k decode 32 long": _case("llama3-2k", "decode", 32, 1003, 7999),
        # prompt batch of the headline benchmark
        "llama-8b prefill 8x512": _case("llama3-8b", "prefill", 8, 512, 512),
        # one long document, close to the longest the model takes
        "llama-8b prefill 7999": _case("llama3-8b", "prefill", 1, 7999, 7999),
        # a few prompts of unequal, odd lengths
        "llama-2k prefill ragged": _case("llama3-2k", "prefill", 6, 37, 1501),
        # continuous batching: prompts in portions beside single tokens
        "llama-2k serve": _case("llama3-2k", "serve", 12, 23, 1201, new=4, budget=1024),
        "nubosun-2k prefill ragged": _case("nubosun-2k", "prefill", 8, 101, 919),
        "nubosun-2k decode 8": _case("nubosun-2k", "decode", 8, 640, 640),
        # replay in full 32 bits, as one checks a checkpoint
        "nubosun-2k float32": _case("nubosun-2k", "prefill", 2, 101, 503, dtype="float32"),
        "bobarax-2k prefill 4096": _case("bobarax-2k", "prefill", 1, 4096, 4096),
    }.items()]


# per model: most tokens of a prompt batch, most rows of a decode step, most cached tokens of all its rows
RANGES = {"llama3-2k": (16000, 64, 128000), "llama3-8b": (8000, 32, 16000), "nubosun-2k": (12000, 32, 40000),
          "bobarax-2k": (12000, 32, 40000)}


def draw(rng):
    def log(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))
    model = rng.choice(list(RANGES))
    tokens, rows_max, cached = RANGES[model]
    kind = rng.choice(("prefill", "decode", "decode", "serve", "prefill"))
    if kind == "decode":
        rows = log(1, rows_max)
        longest = log(32, min(8100, cached // rows))
        return _case(model, kind, rows, rng.randint(max(1, longest // 4), longest), longest)
    if kind == "serve":
        rows = log(2, 16)
        longest = log(32, min(2000, tokens // rows))
        return _case(model, kind, rows, rng.randint(1, longest), longest, new=rng.randint(2, 4), budget=log(64, 2048))
    if model in ("nubosun-2k", "bobarax-2k") and rng.random() < 0.25:
        rows = log(1, 4)
        longest = log(16, 1000 // rows)
        return _case(model, kind, rows, rng.randint(max(1, longest // 4), longest), longest, dtype="float32")
    rows = log(1, 16)
    longest = log(32, min(8100, tokens // rows))
    return _case(model, kind, rows, rng.randint(max(1, longest // 8), longest), longest)


def lengths(case):
    """Prompt lengths, spread evenly between the shortest and the longest."""
    n = case["rows"]
    return [case["longest"]] if n == 1 else [round(case["shortest"] + (case["longest"] - case["shortest"]) * ((i * 5 + 3) % n if n % 5 else i) / (n - 1)) for i in range(n)]


def steps(case):
    """Entries (request, first token, tokens, wanted offsets) of every call, and the requests that end with it."""
    lens = lengths(case)
    if case["kind"] == "prefill":
        return [([(i, 0, n, (n - 1,)) for i, n in enumerate(lens)], list(range(len(lens))))]
    done, out = [0] * len(lens), []
    last = [n + case["new"] - 1 for n in lens]
    while any(d < e for d, e in zip(done, last)):
        entries, room, ends = [], case["budget"], []
        for i, n in enumerate(lens):
            if n <= done[i] < last[i] and room:
                entries.append((i, done[i], 1, (0,)))
                room -= 1
        for i, n in enumerate(lens):
            if done[i] < n and room:
                k = min(room, n - done[i])
                entries.append((i, done[i], k, (k - 1,) if done[i] + k == n else ()))
                room -= k
        for i, _, k, _ in entries:
            done[i] += k
            if done[i] == last[i]:
                ends.append(i)
        out.append((entries, ends))
    return out


class Weights:
    """Random weights under the checkpoint's names, a function of (seed, name); values keep activations near unit size, decays cover many time scales."""

    def __init__(self, cfg, seed, dtype=torch.bfloat16):
        self.cfg, self.seed, self.dtype, self.shapes = cfg, seed, dtype, tensor_shapes(cfg)

    def names(self):
        return self.shapes.keys()

    def get(self, name):
        shape, leaf = self.shapes[name], name.split(".", 1)[-1] if name.startswith("l") else name
        g = torch.Generator(device=DEVICE).manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        n = lambda: torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32)
        u = lambda: torch.rand(shape, generator=g, device=DEVICE, dtype=torch.float32)
        if leaf == "mlp.table":
            f = self.cfg.layers[int(name[1:].split(".")[0])].mlp
            return torch.rand(shape[0], f.experts, generator=g, device=DEVICE).argsort(1)[:, : shape[1]].to(torch.int32)
        if leaf == "mix.A_log":
            t = torch.log(0.5 + 8.0 * u())
        elif leaf == "mix.dt.b":
            t = -4.0 + 3.0 * u()
        elif leaf.startswith("hc") and leaf.endswith(".in"):
            t = 1.0 / shape[0] + 0.1 * n()
        elif leaf.startswith("hc") and leaf.endswith(".mix"):
            t = 0.9 * torch.eye(shape[0], device=DEVICE) + 0.05 * n()
        elif leaf in ("mix.sink", "mix.conv.b"):
            t = 0.5 * n()
        elif leaf.endswith(".bias"):
            t = 0.1 * n()
        elif len(shape) == 1:
            around_zero = isinstance(self.cfg, BobaraxConfig) and "mix." not in leaf
            t = 0.1 * n() + (0.0 if around_zero else 1.0)
        elif "embed" in leaf:
            t = n()
        else:
            t = shape[1] ** -0.5
            if leaf.endswith(("o_proj.weight", "down_proj.weight")) or isinstance(self.cfg, NubosunConfig) and leaf in ("mix.o", "mlp.down"):
                t *= (2 * self.cfg.num_layers) ** -0.5             # what a sublayer adds to the residual stream, as models are initialised
            return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.bfloat16).mul_(t).to(self.dtype)
        return t.to(torch.bfloat16).to(self.dtype)


def _tokens(case, seed):
    """Tokens of every request: its prompt and those that follow it."""
    r = np.random.RandomState(seed % (1 << 31))
    vocab = get_config(case["model"]).vocab_size
    return [r.randint(0, vocab, n + max(1, case["new"])).tolist() for n in lengths(case)]


def prepare(case, seed):
    cfg, lens, dtype = get_config(case["model"]), lengths(case), getattr(torch, case["dtype"])
    toks = _tokens(case, seed)
    eng = Engine(cfg, device=DEVICE, source=Weights(cfg, seed, dtype), dtype=dtype, max_batch=case["rows"], max_seq_len=max(lens) + max(8, case["new"]),
                 prefill_chunk=min(CHUNK, max(case["rows"], case["budget"] or sum(lens))))
    if case["kind"] != "decode":
        calls = [([(i, toks[i][a: a + k], w) for i, a, k, w in entries], ends) for entries, ends in steps(case)]
        return {"engine": eng, "calls": calls}
    eng.prefill([t[:n] for t, n in zip(toks, lens)], 4)
    graph = eng.capture(case["rows"], eng.attn_splits_for(case["rows"], max(lens) + 4), False, io=True)
    eng._load_decode_inputs(case["rows"], [t[n] for t, n in zip(toks, lens)], lens)
    return {"engine": eng, "step": graph, "logits": eng.model.logits[: case["rows"], : cfg.vocab_size]}


def run(state):
    if "step" in state:
        state["step"].replay()
        return state["logits"]
    return [state["engine"].step(entries, end=ends) for entries, ends in state["calls"]]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def work(case):
    cfg, lens, size = get_config(case["model"]), lengths(case), 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "decode":
        calls = [[(i, n, 1, (0,)) for i, n in enumerate(lens)]]
    else:
        calls = [e for e, _ in steps(case)]
    shapes, total, flops = tensor_shapes(cfg), 0.0, 0.0
    product = {k: math.prod(s) for k, s in shapes.items() if len(s) == 2 and not any(x in k for x in ("embed", "head", ".table", ".hc", "conv", "A_log"))}
    head = cfg.vocab_size * cfg.hidden_size
    for entries in calls:
        T, wanted = sum(k for _, _, k, _ in entries), sum(len(w) for _, _, _, w in entries)
        for name, n in product.items():
            share = used = 1.0
            if ".mlp.e" in name:                                   # an expert's matrix: the share of the tokens that meet it, and whether any does
                f = cfg.layers[int(name[1:].split(".")[0])].mlp
                share = f.top / f.experts
                used = 1.0 - (1.0 - share) ** T
            total += size * n * used
            flops += 2.0 * n * T * share
        if wanted:
            total += size * head + (2 if case["kind"] == "decode" and isinstance(cfg, ModelConfig) else 4) * wanted * cfg.vocab_size
            flops += 2.0 * head * wanted
        total += size * T * cfg.hidden_size
        for i in range(cfg.num_layers):
            m = None if not hasattr(cfg, "layers") else cfg.layers[i].mixer
            if isinstance(m, MambaSpec):
                total += 8.0 * len(entries) * m.inner * (m.state + m.conv - 1)
                flops += 7.0 * T * m.inner * m.state
                continue
            if isinstance(m, LightningSpec):
                total += 8.0 * len(entries) * m.heads * m.dim * m.vdim
                flops += 4.0 * T * m.heads * m.dim * m.vdim
                continue
            reach = (lambda p: p + 1) if m is None or not hasattr(m, "chunk") else \
                (lambda p: min(p + 1, m.window)) if m.window else (lambda p: p % m.chunk + 1) if m.chunk else (lambda p: p + 1)
            if m is None:
                row, per_key = 2 * cfg.num_kv_heads * cfg.head_dim, 4.0 * cfg.num_heads * cfg.head_dim
            elif isinstance(cfg, NubosunConfig):
                row, per_key = m.kv_rank + m.rot_dim, 2.0 * m.heads * (m.dim + m.rot_dim + m.vdim)
            else:
                row, per_key = m.kv_heads * (m.dim + m.vdim), 2.0 * m.heads * (m.dim + m.vdim)
            for _, first, k, _ in entries:
                end = first + k
                old = max(0, reach(end - 1) - k) if k < reach(end - 1) else 0          # cached rows of earlier steps that are read
                total += size * row * (k + old)
                flops += per_key * float(sum(reach(p) for p in range(first, end)))
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Errors against 64 bits measured over the listed and some drawn cases: bf16 0.004 (Bobarax) to 0.014 (32 layers with a bf16 residual stream), fp32 2.5e-6.
    Two correct implementations differ by the errors of both; bf16 is given twice what was seen, fp32 four times."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 3e-4}
    return {"rel": 0.03, "max": 0.4}


# ---- the same models in 64 bits ---------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, pos, freq, factor=1.0):
    """x [T, H, D]: dimensions 2i and 2i + 1 of the first 2 len(freq) turned by position * frequency."""
    a = pos[:, None] * freq[None]
    c, s, n = (a.cos() * factor)[:, None], (a.sin() * factor)[:, None], 2 * freq.numel()
    out = x.clone()
    out[..., 0:n:2] = x[..., 0:n:2] * c - x[..., 1:n:2] * s
    out[..., 1:n:2] = x[..., 1:n:2] * c + x[..., 0:n:2] * s
    return out


def _turn_halves(x, pos, freq):
    """x [T, H, D]: dimensions i and i + D / 2 turned together."""
    a = pos[:, None] * freq[None]
    c, s, h = a.cos()[:, None], a.sin()[:, None], x.shape[-1] // 2
    return torch.cat((x[..., :h] * c - x[..., h:] * s, x[..., h:] * c + x[..., :h] * s), -1)


def _attend(q, k, v, scale, visible=None, cap=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] of one sequence; ``visible(i, j)`` beside causality.  Blocks of 1024 queries, one head at a time."""
    T, H, _ = q.shape
    rep, out = H // k.shape[1], torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    j = torch.arange(T, device=q.device)
    for h in range(H):
        kh, vh = k[:, h // rep], v[:, h // rep]
        for a in range(0, T, 1024):
            b = min(T, a + 1024)
            i = torch.arange(a, b, device=q.device)[:, None]
            s = q[a:b, h] @ kh[:b].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            hide = j[None, :b] > i
            if visible is not None:
                hide = hide | ~visible(i, j[None, :b])
            s = s.masked_fill(hide, -math.inf)
            if sink is not None:
                s = torch.cat((s, sink[h].expand(b - a, 1)), 1)
            p = torch.softmax(s, 1)
            out[a:b, h] = p[:, :b] @ vh[:b]
    return out


def _llama(cfg, w, toks, spans, pos, every):
    D, eps, f64 = cfg.head_dim, cfg.rms_eps, torch.float64
    freq = cfg.rope_theta ** (-torch.arange(0, D, 2, dtype=f64, device=DEVICE) / D)
    x = w("model.embed_tokens.weight")[toks]
    for l in range(cfg.num_layers):
        p = f"model.layers.{l}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = (h @ w(p + f"self_attn.{s}_proj.weight").T + (w(p + f"self_attn.{s}_proj.bias") if cfg.qkv_bias else 0.0) for s in "qkv")
        q, k, v = _turn_halves(q.view(-1, cfg.num_heads, D), pos, freq), _turn_halves(k.view(-1, cfg.num_kv_heads, D), pos, freq), v.view(-1, cfg.num_kv_heads, D)
        o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], D ** -0.5) for a, b in spans])
        x = x + o.reshape(x.shape[0], -1) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        x = x + (F.silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    return _rms(x[every], eps) * w("model.norm.weight") @ w("lm_head.weight").T


def _yarn(rot):
    """Frequencies and the factor on cos and sin, for base / dims / YaRN scaling."""
    f, factor = [], 1.0
    lo = hi = 0.0
    sc = rot.scaling
    if sc:
        at = lambda turns: rot.dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot.base))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), rot.dims - 1)
        factor = 0.1 * math.log(sc["factor"]) + 1.0
    for i in range(rot.dims // 2):
        v = rot.base ** (-2.0 * i / rot.dims)
        if sc:
            r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            v = v / sc["factor"] * r + v * (1.0 - r)
        f.append(v)
    return torch.tensor(f, dtype=torch.float64, device=DEVICE), factor


def _mamba(h, w, p, m, spans):
    x, z = (h @ w(p + "in").T).split(m.inner, 1)
    taps, bias, rate, ys = w(p + "conv"), w(p + "conv.b"), -torch.exp(w(p + "A_log")), []
    wx, wdt, bdt, d = w(p + "x"), w(p + "dt"), w(p + "dt.b"), w(p + "D")
    # all sequences side by side, the shorter ones filled up with zeros behind their end
    L = max(b - a for a, b in spans)
    u = torch.zeros(len(spans), L, m.inner, dtype=h.dtype, device=DEVICE)
    for s, (a, b) in enumerate(spans):
        u[s, : b - a] = F.silu(F.conv1d(F.pad(x[a:b].T, (m.conv - 1, 0))[None], taps[:, None], bias, groups=m.inner)[0].T)
    proj = u @ wx.T
    dt = F.softplus(proj[..., : m.dt_rank] @ wdt.T + bdt)
    B, C = proj[..., m.dt_rank: m.dt_rank + m.state], proj[..., m.dt_rank + m.state:]
    state, y = torch.zeros(len(spans), m.inner, m.state, dtype=h.dtype, device=DEVICE), torch.empty_like(u)
    for t in range(L):
        state = torch.exp(dt[:, t, :, None] * rate) * state + (dt[:, t] * u[:, t])[..., None] * B[:, t, None]
        y[:, t] = (state @ C[:, t, :, None])[..., 0] + d * u[:, t]
    y = torch.cat([y[s, : b - a] for s, (a, b) in enumerate(spans)])
    return (y * F.silu(z)) @ w(p + "o").T


def _nubosun(cfg, w, toks, spans, pos, every):
    eps, T = cfg.rms_eps, toks.numel()
    xs = [w("embed")[toks] * cfg.embedding_scale for _ in range(cfg.streams)]

    def sublayer(xs, fn, p, n):
        hin, hout, mix = w(f"{p}hc{n}.in"), w(f"{p}hc{n}.out"), w(f"{p}hc{n}.mix")
        y = fn(_rms(sum(hin[s] * x for s, x in enumerate(xs)), eps) * w(f"{p}norm{n}")) * w(f"{p}ls{n}")
        return [sum(mix[s, t] * x for s, x in enumerate(xs)) + hout[t] * y for t in range(cfg.streams)]

    def latent(h, p, m):
        freq, factor = _yarn(m.rot)
        q = (h @ w(p + "q").T).view(T, m.heads, m.dim + m.rot_dim)
        kv = h @ w(p + "dkv").T
        c = _rms(kv[:, : m.kv_rank], eps) * w(p + "dkv.norm")
        k = torch.cat(((c @ w(p + "uk").T).view(T, m.heads, m.dim), _turn(kv[:, None, m.kv_rank:], pos, freq, factor).expand(T, m.heads, m.rot_dim)), 2)
        q = torch.cat((q[..., : m.dim], _turn(q[..., m.dim:], pos, freq, factor)), 2)
        v, sink = (c @ w(p + "uv").T).view(T, m.heads, m.vdim), w(p + "sink")
        o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], m.scale, sink=sink) for a, b in spans])
        return o.reshape(T, -1) @ w(p + "o").T

    def mlp(h, p, f):
        g, u = (h @ w(p + "gate").T).clamp(max=f.limit), (h @ w(p + "up").T).clamp(-f.limit, f.limit)
        return (g * torch.sigmoid(f.slope * g) * (u + 1.0)) @ w(p + "down").T

    for i in cfg.runs:
        lay, p = cfg.layers[i], f"l{i}."
        mixer = (lambda h: _mamba(h, w, p + "mix.", lay.mixer, spans)) if isinstance(lay.mixer, MambaSpec) else (lambda h: latent(h, p + "mix.", lay.mixer))
        xs = sublayer(xs, mixer, p, 1)
        if lay.mlp is not None:
            xs = sublayer(xs, lambda h: mlp(h, p + "mlp.", lay.mlp), p, 2)
    logits = _rms(sum(xs)[every], eps) * w("final.norm") @ w("head").T
    return cfg.logit_softcap * torch.tanh(logits / cfg.logit_softcap) if cfg.logit_softcap else logits


def _bobarax(cfg, w, toks, spans, pos, every):
    eps, T, kv = cfg.rms_eps, toks.numel(), {}
    norm = lambda x, name: _rms(x, eps) * (1.0 + w(name))

    def lightning(h, p, m):
        q, k, v = (F.silu(h @ w(p + s).T).view(T, m.heads, -1) for s in "qkv")
        o = torch.empty_like(v)
        for a, b in spans:
            j = torch.arange(b - a, device=DEVICE)
            for hd in range(m.heads):
                for c in range(0, b - a, 1024):
                    e = min(b - a, c + 1024)
                    far = (j[c:e, None] - j[None, :e]).to(torch.float64)
                    power = torch.where(far >= 0, torch.exp(math.log(m.decay[hd]) * far.clamp(min=0)), torch.zeros_like(far))
                    o[a + c: a + e, hd] = (q[a + c: a + e, hd] @ k[a: a + e, hd].T * power) @ v[a: a + e, hd]
        return (_rms(o.reshape(T, -1), eps) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T

    def attention(h, i, p, m):
        freq = m.rot.base ** (-2.0 * torch.arange(m.rot.dims // 2, dtype=torch.float64, device=DEVICE) / m.rot.dims) if m.rot else None
        turn = (lambda x: _turn(x, pos, freq)) if m.rot else (lambda x: x)
        whole = lambda s, n: turn((_rms(h @ w(p + s).T, eps) * w(p + s + ".norm")).view(T, n, m.dim))
        q = whole("q", m.heads)
        kv[i] = (whole("k", m.kv_heads), (h @ w(p + "v").T).view(T, m.kv_heads, m.vdim)) if m.kv_from is None else kv[m.kv_from]
        see = (lambda a, b: a - b < m.window) if m.window else (lambda a, b: a // m.chunk == b // m.chunk) if m.chunk else None
        o = torch.cat([_attend(q[a:b], kv[i][0][a:b], kv[i][1][a:b], m.scale, see, m.softcap) for a, b in spans]).reshape(T, -1)
        return (o * torch.sigmoid(h @ w(p + "g").T) if m.gated else o) @ w(p + "o").T

    def mlp(h, p, f):
        if not isinstance(f, TableMoeSpec):
            return (torch.relu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T
        y, chosen = torch.zeros_like(h), w.plain(p + "table")[toks].long()
        for e in range(f.experts):
            r = (chosen == e).any(1).nonzero()[:, 0]
            g, u = (h[r] @ w(f"{p}e{e}.gate").T).clamp(max=f.limit), (h[r] @ w(f"{p}e{e}.up").T).clamp(-f.limit, f.limit)
            y[r] += (g * torch.sigmoid(f.slope * g) * (u + 1.0)) @ w(f"{p}e{e}.down").T / f.top
        return y

    x = w("embed")[toks]
    for i, lay in enumerate(cfg.layers):
        p, m = f"l{i}.", lay.mixer
        h = norm(x, p + "norm1")
        y = lightning(h, p + "mix.", m) if isinstance(m, LightningSpec) else attention(h, i, p + "mix.", m)
        x = x + cfg.residual_mult * norm(y, p + "norm1b")
        if lay.mlp is not None:
            x = x + cfg.residual_mult * norm(mlp(norm(x, p + "norm2"), p + "mlp.", lay.mlp), p + "norm2b")
    return norm(x[every], "final.norm") @ w("embed").T * cfg.logit_scale


class _Wide:
    """Weights in 64 bits, by name."""

    def __init__(self, weights):
        self.plain = weights.get

    def __call__(self, name):
        return self.plain(name).to(torch.float64)


def exact(case, seed):
    cfg, lens, toks = get_config(case["model"]), lengths(case), _tokens(case, seed)
    decode = case["kind"] == "decode"
    calls = [([(i, n, 1, (0,)) for i, n in enumerate(lens)], ())] if decode else steps(case)
    total = [n + (1 if decode else max(0, case["new"] - 1)) for n in lens]
    start = np.concatenate(([0], np.cumsum(total)))
    ids = torch.tensor([t for ts, n in zip(toks, total) for t in ts[:n]], device=DEVICE)
    pos = torch.cat([torch.arange(n, dtype=torch.float64, device=DEVICE) for n in total])
    want = [[int(start[i]) + first + o for i, first, _, w in entries for o in w] for entries, _ in calls]
    fn = _nubosun if isinstance(cfg, NubosunConfig) else _bobarax if isinstance(cfg, BobaraxConfig) else _llama
    every = torch.tensor([r for rows in want for r in rows], device=DEVICE)
    with torch.no_grad():
        logits = fn(cfg, _Wide(Weights(cfg, seed)), ids, list(zip(start[:-1].tolist(), start[1:].tolist())), pos, every)
    return logits if decode else list(logits.split([len(rows) for rows in want]))
