"""Serving work measured on one GPU: prompts go in, given tokens follow one by one, logits and the cache come out.

A pass is what a serving program does with a batch from its first token to its last: ``Engine.start_batch``, ``Engine.prefill`` (or
portions through ``Engine.step``), ``Engine.step_from_host`` for every given token, ``Engine.step`` for the last one, whose logits it
reads.  The tokens are given, not sampled, so that the logits of two implementations are those of the same sequence.  The models are
this framework's four kinds at the widths of its presets and benchmarks, with fewer layers and random weights.  As in trained
models a layer adds little to the residual stream (output matrices scaled by depth) and routers are decisive, so that a
last bit somewhere does not send a token to an expert of equal weight."""
from __future__ import annotations

import math
import zlib
from dataclasses import replace

import torch

from mojo_linuxperiments_b200.engine.engine import Engine
from mojo_linuxperiments_b200.models import config as C
from mojo_linuxperiments_b200.models import layered_config as LC
from mojo_linuxperiments_b200.models import layered_weights as LW
from mojo_linuxperiments_b200.models.weights import LinearW

DEVICE = "cuda"
BF = torch.bfloat16
ROUTER_GAIN = 3.0        # standard deviation of router logits
VOCAB = 32000


# ---- models -------------------------------------------------------------------------------------------------------------------
def config(model: str):
    if model == "llama":            # W8A8, dense: the width of the 8B shape
        return replace(C.llama3_8b(), n_layers=4, vocab=VOCAB)
    if model == "qwen":             # W8A8, mixture: the width of the 30B shape, 128 experts of which 8 are active
        return replace(C.qwen3_30b_a3b(), n_layers=4, vocab=VOCAB)
    if model == "volonex":          # bf16, chunked attention with sinks; the chunk is short enough to matter in a prompt
        return LC.volonex(2048, 8, 16, 8, 8192, VOCAB, chunk=512)
    if model == "volonex32":        # the same design with everything in 32 bits, as a trace is replayed
        return LC.volonex(2048, 3, 16, 8, 8192, VOCAB, chunk=512)
    if model == "rakelorn":         # bf16, latent attention, recurrent layers, mixture
        return replace(LC.rakelorn_2b(), layers=LC.rakelorn_2b().layers[:6], vocab=VOCAB)
    raise ValueError(model)


def element(model: str) -> str:
    return "float32" if model == "volonex32" else "bfloat16"


def generator(seed: int, name: str) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed((seed * 0x9E3779B1 + zlib.crc32(name.encode())) & 0x7FFFFFFF)


def w8a8_weights(cfg, seed: int) -> dict:
    """Device weights of a W8A8 model: int8 matrices with a scale per channel, everything else bf16."""
    d, hd, E, depth = cfg.d_model, cfg.head_dim, cfg.n_experts, (2 * cfg.n_layers) ** -0.5

    def linear(name, n, k, gain=1.0, lead=()):
        g = generator(seed, name)
        q = torch.randint(-127, 128, lead + (n, k), dtype=torch.int8, device=DEVICE, generator=g)
        s = (torch.rand(lead + (n,), device=DEVICE, generator=g) * 0.5 + 0.75) * (gain * k ** -0.5 / 73.3)
        return LinearW(q, s)

    def gain(name, n):
        return (1.0 + 0.1 * torch.randn((n,), device=DEVICE, generator=generator(seed, name))).to(BF)

    w = {"embed": torch.randn((cfg.vocab, d), device=DEVICE, generator=generator(seed, "embed"), dtype=BF), "final_norm": gain("final", d),
         "lm_head": linear("head", cfg.vocab, d), "vocab_offset": 0, "layers": []}
    for l in range(cfg.n_layers):
        L = {"attn_norm": gain(f"{l}an", d), "mlp_norm": gain(f"{l}mn", d),
             "qkv": linear(f"{l}qkv", (cfg.n_heads + 2 * cfg.n_kv_heads) * hd, d), "o": linear(f"{l}o", d, cfg.n_heads * hd, depth)}
        if cfg.qk_norm:
            L["q_norm"], L["k_norm"] = gain(f"{l}qn", hd), gain(f"{l}kn", hd)
        if E:
            L["router"] = linear(f"{l}r", E, d, ROUTER_GAIN)
            L["experts_gate_up"] = linear(f"{l}gu", 2 * cfg.moe_ffn, d, lead=(E,))
            L["experts_down"] = linear(f"{l}dn", d, cfg.moe_ffn, depth, lead=(E,))
        else:
            L["gate_up"] = linear(f"{l}gu", 2 * cfg.ffn, d)
            L["down"] = linear(f"{l}dn", d, cfg.ffn, depth)
        w["layers"].append(L)
    return w


class Tensors:
    """Checkpoint tensors of a layer-by-layer model by name, made on the device when they are asked for."""

    def __init__(self, cfg, seed: int):
        self.shapes, self.seed, self.depth = LW.tensor_shapes(cfg), seed, (2 * len(cfg.layers)) ** -0.5

    def __getitem__(self, name: str) -> torch.Tensor:
        role, shape = self.shapes[name]
        g = generator(self.seed, name)
        if role == "matrix":
            n = torch.randn(shape, generator=g, device=DEVICE, dtype=BF)
            gain = ROUTER_GAIN if name.endswith("router") else self.depth if name.endswith((".o", ".down")) else 1.0
            return n if name == "embed" else n.mul_(gain * shape[1] ** -0.5)
        if role == "shift":
            return torch.rand(shape, generator=g, device=DEVICE).to(BF)
        n = torch.randn(shape, generator=g, device=DEVICE)
        return {"alpha": 0.5 + 0.05 * n, "gain": 1 + 0.1 * n, "bias": 0.1 * n, "sink": n, "step": n, "correction": 0.01 * n}[role].to(BF)


# ---- cases --------------------------------------------------------------------------------------------------------------------
# ``prompt``: tokens per sequence (ragged: a quarter of that up to that), ``steps``: given tokens after it, one by one
# ``turns``: the prompt comes in that many portions
def listed():
    return [
        # one user, a short question: launches and latencies of a decode step at batch 1
        case("llama", 1, 33, 32, "llama_chat_1x33"),
        # time to first token of one prompt of the benchmark's length
        case("llama", 1, 1024, 0, "llama_prompt_1x1024"),
        # the benchmark's batch: its decode steps over a short context
        case("llama", 32, 200, 64, "llama_batch_32x200"),
        # documents read in bulk: the largest prefill call
        case("llama", 32, 1024, 0, "llama_prompts_32x1024"),
        # few long sequences of odd length: attention over long caches
        case("llama", 3, 3001, 24, "llama_long_3x3001"),
        # a wide batch, above the 64 tokens up to which the decode linears stream weights
        case("llama", 100, 64, 32, "llama_wide_100x64"),
        # prompts of different lengths in one call
        case("llama", 7, 777, 16, "llama_ragged_7x777", ragged=True),
        # mixture of experts: a batch that decodes, and prompts
        case("qwen", 16, 150, 48, "qwen_batch_16x150"),
        case("qwen", 8, 1000, 4, "qwen_prompts_8x1000"),
        # unquantised model, the prompt in two portions
        case("volonex", 12, 700, 32, "volonex_batch_12x700", turns=2),
        # a trace in 32 bits
        case("volonex32", 2, 190, 8, "volonex_trace_2x190"),
        # latent attention, recurrence, mixture
        case("rakelorn", 8, 500, 32, "rakelorn_batch_8x500"),
    ]


def case(model, batch, prompt, steps, name=None, ragged=False, turns=1):
    c = {"model": model, "batch": batch, "prompt": prompt, "steps": steps, "ragged": ragged, "turns": turns}
    return {"name": name, **c} if name else c


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["llama", "llama", "llama", "llama", "qwen", "qwen", "volonex", "volonex", "volonex32", "rakelorn"])
    if model == "volonex32":
        return case(model, rng.randint(1, 2), log(16, 190), rng.randint(0, 8), turns=rng.randint(1, 2))
    tokens = {"llama": 16000, "qwen": 8000, "volonex": 8400, "rakelorn": 4000}[model]
    batch = log(1, 100)
    prompt = log(16, max(32, min(3001, tokens // batch)))
    return case(model, batch, prompt, rng.choice([0, rng.randint(1, 32), rng.randint(8, 32)]), ragged=batch > 1 and rng.random() < 0.3,
                turns=rng.randint(1, 2) if model == "volonex" else 1)


def lengths(c, seed: int) -> list[int]:
    B, S = c["batch"], c["prompt"]
    if not c["ragged"]:
        return [S] * B
    u = torch.rand(B, generator=torch.Generator().manual_seed(seed + 77)).tolist()
    return [max(1, int(S * (0.25 + 0.75 * v))) for v in u]


def token_ids(c, cfg, seed: int):
    """(prompt of every sequence, given tokens [steps, batch]) on the host."""
    g = torch.Generator().manual_seed(seed + 1)
    prompts = [torch.randint(0, cfg.vocab, (n,), generator=g) for n in lengths(c, seed)]
    return prompts, torch.randint(0, cfg.vocab, (c["steps"], c["batch"]), generator=g)


def prepare(c, seed: int):
    cfg = config(c["model"])
    prompts, given = token_ids(c, cfg, seed)
    total = c["prompt"] + c["steps"] + 1
    rt = C.RuntimeConfig(max_batch=c["batch"], max_seq_len=-(-total // 128) * 128, dtype=element(c["model"]))
    if isinstance(cfg, C.ModelConfig):
        weights = w8a8_weights(cfg, seed)
    else:
        weights = LW.place(cfg, rt, Tensors(cfg, seed), torch.device(DEVICE))
    return {"engine": Engine(cfg, rt, weights=weights), "case": c, "total": total, "given": given.pin_memory() if c["steps"] else given,
            "prompts": prompts if c["ragged"] or c["turns"] > 1 else torch.stack(prompts).pin_memory(),
            "sampled": torch.empty(c["batch"], dtype=torch.int64).pin_memory()}


def run(state):
    eng, c, given = state["engine"], state["case"], state["given"]
    B, turns = c["batch"], c["turns"]
    eng.start_batch(B, state["total"])
    if turns > 1:
        parts = [torch.tensor_split(p, turns) for p in state["prompts"]]
        for t in range(turns):
            entries = [(b, p[t], [p[t].numel() - 1] if t == turns - 1 else []) for b, p in enumerate(parts) if p[t].numel()]
            logits = eng.step(entries)
        logits = torch.cat(logits)
    else:
        eng.prefill(state["prompts"])
        logits = eng.model.last_logits
    for t in range(c["steps"] - 1):
        eng.step_from_host(given[t], state["sampled"])
    if c["steps"]:
        logits = torch.cat(eng.step([(b, given[-1, b:b + 1], [0]) for b in range(B)]))
    return {"logits": logits, "cache": eng.kv.storage}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------
def parameters(cfg):
    """(elements every token multiplies in the layers, elements of one expert of all layers, experts, chosen, pairs of one
    (query, key): multiplications per layer stack, cached elements per token), without embedding and head."""
    if isinstance(cfg, C.ModelConfig):
        d, hd, n = cfg.d_model, cfg.head_dim, cfg.n_layers
        dense = n * (d * (cfg.n_heads + 2 * cfg.n_kv_heads) * hd + cfg.n_heads * hd * d)
        dense += n * (cfg.n_experts * d if cfg.is_moe else 3 * d * cfg.ffn)
        return dense, n * 3 * d * cfg.moe_ffn, cfg.n_experts, cfg.top_k, n * 2 * cfg.n_heads * hd, n * 2 * cfg.n_kv_heads * hd
    dense = expert = experts = top = pair = cached = 0
    d = cfg.d_model
    for l in cfg.layers:
        m = l.mixer
        dense += m.matrix_elements(d)
        if isinstance(m, LC.AttentionSpec):
            pair += m.heads * (m.dim + m.vdim)
            cached += m.kv_heads * (m.dim + m.vdim)
        elif isinstance(m, LC.LatentSpec):
            pair += m.heads * (m.dim + m.rot_dim + m.vdim)
            cached += m.kv_rank + m.rot_dim
        if isinstance(l.mlp, LC.MoE):
            dense += d * l.mlp.outputs
            expert, experts, top = expert + 2 * d * l.mlp.ff, l.mlp.experts, l.mlp.top
        elif l.mlp is not None:
            dense += l.mlp.matrix_elements(d)
    return dense, expert, experts, top, pair, cached


def work(c):
    """Every forward pass reads the weights that its tokens use, every token writes its cache rows, every decoded token
    reads those of its sequence, every call writes logits."""
    cfg = config(c["model"])
    dense, expert, experts, top, pair, cached = parameters(cfg)
    quantised = isinstance(cfg, C.ModelConfig)
    elem = 1 if quantised else 4 if element(c["model"]) == "float32" else 2
    kv = 4 if element(c["model"]) == "float32" else 2
    chunk = next((l.mixer.chunk for l in cfg.layers if isinstance(l.mixer, LC.AttentionSpec)), None) if not quantised else None
    S = c["prompt"] * (0.625 if c["ragged"] else 1.0)
    B, T = c["batch"], c["steps"]

    def weights(tokens):
        used = experts * (1.0 - (1.0 - top / experts) ** tokens) if experts else 0
        return (dense + expert * used + cfg.vocab * cfg.d_model) * elem

    def visible(position):
        return position % chunk + 1 if chunk else position + 1

    logits = B * cfg.vocab * (2 if quantised else 4)
    bytes_ = weights(B * S) + B * (S + T) * cached * kv + logits * (1 + T)
    flops = 2.0 * B * (S + T) * (dense + expert * top) + 2.0 * B * (1 + T) * cfg.vocab * cfg.d_model
    full, rest = (int(S) // chunk, int(S) % chunk) if chunk else (0, S)
    flops += 2.0 * B * pair * (full * (chunk or 0) ** 2 / 2 + rest ** 2 / 2)
    for t in range(T):
        seen = visible(int(S) + t)
        bytes_ += weights(B) + B * seen * cached * kv
        flops += 2.0 * B * pair * seen
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(c):
    # int8 rows and bf16 tensors between the kernels: a last bit moves other values across an edge, which then differ by a step
    # (the forms of decode attention that this framework has differ by 0.009 to 0.013, each is 0.016 from 64 bits); bf16 alone
    # is 0.002 to 0.006 from 64 bits, the 32-bit form 1e-6
    return {"llama": {"rel": 0.03, "max": 0.6}, "qwen": {"rel": 0.03}, "volonex": {"rel": 0.01}, "rakelorn": {"rel": 0.02},
            "volonex32": {"rel": 1e-5}}[c["model"]]


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------
def softmax_attention(q, k, v, visible, sink=None):
    """q [T, H, a], k [T, H, a], v [T, H, b] with scaled queries -> [T, H, b], a few heads at a time."""
    out = torch.empty(q.shape[:2] + v.shape[2:], dtype=q.dtype, device=q.device)
    for h in range(0, q.shape[1], 8):
        s = torch.einsum("ihd,jhd->hij", q[:, h:h + 8], k[:, h:h + 8]).masked_fill(~visible, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[h:h + 8, None, None])
        e = (s - top).exp()
        total = e.sum(-1, keepdim=True)
        if sink is not None:
            total = total + (sink[h:h + 8, None, None] - top).exp()
        out[:, h:h + 8] = torch.einsum("hij,jhd->ihd", e / total, v[:, h:h + 8])
    return out


def causal(T, chunk=None):
    i = torch.arange(T, device=DEVICE)
    seen = i[None] <= i[:, None]
    return seen & (i[None] // chunk == i[:, None] // chunk) if chunk else seen


def per_sequence(lens, fn, *rows):
    return torch.cat([fn(*parts) for parts in zip(*(r.split(lens) for r in rows))])


def rms(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def hadamard():
    h = torch.ones((1, 1), dtype=torch.float64, device=DEVICE)
    while h.shape[0] < 128:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)])
    return h * 128 ** -0.5


def exact_w8a8(cfg, seed, ids, lens):
    W = w8a8_weights(cfg, seed)
    had, hd, H, G, D = hadamard(), cfg.head_dim, cfg.n_heads, cfg.n_kv_heads, torch.float64
    pos = torch.cat([torch.arange(n, device=DEVICE) for n in lens]).to(D)
    ang = pos[:, None] * float(cfg.rope_theta) ** (-torch.arange(0, hd, 2, dtype=D, device=DEVICE) / hd)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rows(x):            # what a quantised linear reads: rotated rows as whole numbers, and their scale
        x = (x.view(-1, x.shape[1] // 128, 128) @ had).view(x.shape)
        s = x.abs().amax(-1, keepdim=True) / 127
        return (x / s).round(), s

    def linear(xs, q, scale):
        return xs[0] @ q.to(D).t() * xs[1] * scale.to(D)

    def turn(x):
        a, b = x.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def swiglu(gu):
        g, u = gu.chunk(2, -1)
        return g.mul_(torch.sigmoid(g)).mul_(u)

    def attend(q, k, v):
        return softmax_attention(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), causal(q.shape[0])).flatten(1)

    h = W["embed"][ids].to(D)
    for L in W["layers"]:
        qkv = linear(rows(rms(h, cfg.eps) * L["attn_norm"].to(D)), L["qkv"].qweight, L["qkv"].scale).view(-1, H + 2 * G, hd)
        q, k, v = qkv.split([H, G, G], 1)
        if cfg.qk_norm:
            q, k = rms(q, cfg.eps) * L["q_norm"].to(D), rms(k, cfg.eps) * L["k_norm"].to(D)
        a = per_sequence(lens, attend, turn(q) * hd ** -0.5, turn(k), v)
        h = h + linear(rows(a), L["o"].qweight, L["o"].scale)
        xs = rows(rms(h, cfg.eps) * L["mlp_norm"].to(D))
        if not cfg.is_moe:
            h = h + linear(rows(swiglu(linear(xs, L["gate_up"].qweight, L["gate_up"].scale))), L["down"].qweight, L["down"].scale)
            continue
        p, chosen = linear(xs, L["router"].qweight, L["router"].scale).softmax(-1).topk(cfg.top_k, -1)
        p = p / p.sum(-1, keepdim=True) if cfg.norm_topk_prob else p
        for e in range(cfg.n_experts):
            at, k = (chosen == e).nonzero(as_tuple=True)
            if at.numel():
                gu = linear((xs[0][at], xs[1][at]), L["experts_gate_up"].qweight[e], L["experts_gate_up"].scale[e])
                h[at] += p[at, k, None] * linear(rows(swiglu(gu)), L["experts_down"].qweight[e], L["experts_down"].scale[e])
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    return linear(rows(rms(h[last], cfg.eps) * W["final_norm"].to(D)), W["lm_head"].qweight, W["lm_head"].scale)


def turn_pairs(x, pos, rot):
    """Neighbouring pairs of the first ``rot.dims`` of x [T, heads, dim] turn with the position, slower ones scaled (YaRN)."""
    n, y = rot.dims, rot.scaling
    freq, mag = float(rot.base) ** (-torch.arange(0, n, 2, dtype=torch.float64, device=DEVICE) / n), 1.0
    if y is not None:
        at = [n * math.log(y.original / (2 * math.pi * r)) / (2 * math.log(rot.base)) for r in (y.fast, y.slow)]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), n - 1)
        ramp = ((torch.arange(n // 2, device=DEVICE, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        freq, mag = freq * (1 - ramp) + freq / y.factor * ramp, 0.1 * math.log(y.factor) + 1
    ang = (pos[:, None] * freq)[:, None]
    c, s, out = ang.cos() * mag, ang.sin() * mag, x.clone()
    a, b = x[..., 0:n:2], x[..., 1:n:2]
    out[..., 0:n:2], out[..., 1:n:2] = a * c - b * s, b * c + a * s
    return out


def exact_layered(cfg, seed, ids, lens):
    names, D = Tensors(cfg, seed), torch.float64

    def t(name):
        return names[name].to(D)

    def norm(name, x):
        if cfg.design.norm == "scalar_rms":
            return rms(x, cfg.eps) * t(name)
        return torch.tanh(t(name + ".alpha") * x) * t(name) + t(name + ".b")

    pos = torch.cat([torch.arange(n, device=DEVICE) for n in lens]).to(D)

    def attention(h, p, m):
        q, k = ((h @ t(p + n).t()).view(-1, heads, m.dim) for n, heads in (("q", m.heads), ("k", m.kv_heads)))
        v = (h @ t(p + "v").t()).view(-1, m.kv_heads, m.vdim)
        if m.rot is not None:
            q, k = turn_pairs(q, pos, m.rot), turn_pairs(k, pos, m.rot)
        k, v, sink = k.repeat_interleave(m.heads // m.kv_heads, 1), v.repeat_interleave(m.heads // m.kv_heads, 1), t(p + "sink")
        o = per_sequence(lens, lambda q, k, v: softmax_attention(q, k, v, causal(q.shape[0], m.chunk), sink), q * m.scale, k, v)
        return (o * torch.sigmoid(h @ t(p + "g").t())[:, :, None]).flatten(1)

    def latent(h, p, m):
        q = (rms(h @ t(p + "dq").t(), cfg.eps) * t(p + "dq.norm") @ t(p + "uq").t()).view(-1, m.heads, m.dim + m.rot_dim)
        c, kr = (h @ t(p + "dkv").t()).split([m.kv_rank, m.rot_dim], -1)
        c = rms(c, cfg.eps) * t(p + "dkv.norm")
        q = torch.cat([q[..., :m.dim], turn_pairs(q[..., m.dim:], pos, m.rot)], -1)
        kr = turn_pairs(kr[:, None], pos, m.rot).expand(-1, m.heads, -1)
        k, v = torch.cat([(c @ t(p + "uk").t()).view(-1, m.heads, m.dim), kr], -1), (c @ t(p + "uv").t()).view(-1, m.heads, m.vdim)
        o = per_sequence(lens, lambda q, k, v: softmax_attention(q, k, v, causal(q.shape[0])), q * m.scale, k, v)
        return (o * torch.sigmoid(h @ t(p + "g").t())[:, :, None]).flatten(1)

    def recurrent(h, p, m):
        z, u = (h @ t(p + n).t() + t(p + n + ".b") for n in "zx")
        z, g = torch.sigmoid(z), h @ t(p + "g").t()
        u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        keep, new, state = 1 - z, z * u, torch.empty_like(z)
        starts, lefts = torch.tensor([0] + lens[:-1], device=DEVICE).cumsum(0), torch.tensor(lens, device=DEVICE)
        s = torch.zeros((len(lens), z.shape[1]), dtype=D, device=DEVICE)
        for i in range(max(lens)):                 # one position of all sequences at a time
            at = starts + torch.minimum(lefts - 1, torch.full_like(lefts, i))
            s = torch.where((lefts > i)[:, None], keep[at] * s + new[at], s)
            state[at] = s
        return state * (g * torch.sigmoid(g))

    def feed_forward(h, p, f):
        if isinstance(f, LC.GatedMLP):
            g, u = (h @ t(p + "gate").t()).clamp(max=f.limit), (h @ t(p + "up").t()).clamp(-f.limit, f.limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ t(p + "down").t()
        s = (h @ t(p + "router").t()).softmax(-1)
        choice = s + t(p + "correction")
        best = choice.view(-1, f.groups, f.outputs // f.groups).amax(-1).topk(f.keep, -1).indices
        open_ = torch.zeros((h.shape[0], f.groups), dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
        chosen = choice.masked_fill(~open_.repeat_interleave(f.outputs // f.groups, 1), -math.inf).topk(f.top, -1).indices
        w, out = s.gather(1, chosen) * f.scale, torch.zeros_like(h)
        for e in range(f.outputs):
            at, k = (chosen == e).nonzero(as_tuple=True)
            if at.numel():
                y = torch.relu(h[at] @ t(f"{p}e{e}.up").t()).pow(2) @ t(f"{p}e{e}.down").t() if e < f.experts else h[at]
                out[at] += w[at, k, None] * y
        return out

    mix = {"attention": attention, "latent_attention": latent, "mingru": recurrent}
    x = t("embed")[ids] * cfg.embed_scale
    for i, l in enumerate(cfg.layers):
        h = norm(f"l{i}.norm1", x)
        if cfg.design.token_shift:
            before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
            before[pos == 0] = 0
            h = h + t(f"l{i}.shift") * (before - h)
        x = x + cfg.residual_mult * (mix[l.mixer.kind](h, f"l{i}.mix.", l.mixer) @ t(f"l{i}.mix.o").t())
        if l.mlp is not None:
            x = x + cfg.residual_mult * feed_forward(norm(f"l{i}.norm2", x), f"l{i}.mlp.", l.mlp)
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    return norm("final.norm", x[last]) @ t("head").t()


def exact(c, seed: int):
    cfg = config(c["model"])
    prompts, given = token_ids(c, cfg, seed)
    ids = torch.cat([torch.cat([p, given[:, b]]) for b, p in enumerate(prompts)]).to(DEVICE)
    lens = [p.numel() + c["steps"] for p in prompts]
    fn = exact_w8a8 if isinstance(cfg, C.ModelConfig) else exact_layered
    with torch.no_grad():
        return {"logits": fn(cfg, seed, ids, lens), "cache": None}
