"""Workloads that stand for how the serving framework is used, for measuring it and comparing its outputs.

A pass is one step of an external scheduler through `GenerationEngine.run_step`: whole prompts ("prefill"), one new token for
every open sequence ("decode"), or a new prompt beside sequences that go on ("mixed", continuous batching).  The models have
the layer sizes, heads, experts and vocabularies of the framework's own configurations and fewer layers (all layers of a kind
cost the same), random weights and uniform random tokens.

    listed()              named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   model, engine, token ids and open sequences, on the GPU
    run(state)            one pass; returns logits
    work(case)            bytes and operations that a pass cannot do without
    tolerance(case)       how far another correct implementation may be off
    exact(case, seed)     what `run` returns, in 64 bits, by plain torch
"""

import math
import random

import torch
import torch.nn.functional as F

from nkipy_b200.models import config as C
from nkipy_b200.models import registry
from nkipy_b200.models.engine import GenerationEngine, StepEntry

DEV = "cuda"
CHUNK = 16384                            # tokens of a prefill step: the engine's default

# the framework's configurations at a reduced depth; gpt-oss and redodra keep a whole period of their layer kinds
CONFIGS = {
    "llama": lambda: C.llama3_8b(num_layers=4),
    "qwen3": lambda: C.qwen3_30b_a3b(num_layers=4),
    "gpt-oss": lambda: C.gpt_oss_20b(num_layers=4),
    "redodra": lambda: C.redodra_shape(4096, layers=5, heads=32, kv_heads=8, ff=14336),
}


def case_of(model, mode, batch, length, ragged=False, portion=0, dtype="bfloat16", **name):
    """batch sequences of `length` tokens (ragged: unequal, down to half of it); portion: tokens of the prompt that arrives in
    a mixed step."""
    return dict(model=model, mode=mode, batch=batch, length=length, ragged=ragged, portion=portion, dtype=dtype, **name)


def listed():
    return [
        # one user's chat: latency of a token
        case_of("llama", "decode", 1, 203, name="llama-decode-1"),
        # the serving benchmark: 64 sequences of 1024 tokens
        case_of("llama", "decode", 64, 1024, name="llama-decode-64"),
        # a few long documents: reading the cache counts as much as the weights
        case_of("llama", "decode", 7, 7000, True, name="llama-decode-long"),
        # time to the first token of one short prompt
        case_of("llama", "prefill", 1, 77, name="llama-prefill-short"),
        # a full prefill step of the serving benchmark, the largest
        case_of("llama", "prefill", 16, 1024, name="llama-prefill-full"),
        # continuous batching: a prompt joins sequences that go on decoding
        case_of("llama", "mixed", 24, 600, True, portion=390, name="llama-mixed"),
        # mixture of experts, the serving benchmark's second half
        case_of("qwen3", "decode", 128, 512, name="qwen3-decode-128"),
        # prompts of unequal lengths through routed experts
        case_of("qwen3", "prefill", 5, 900, True, name="qwen3-prefill-ragged"),
        # batch 1 with sinks, windows and biases
        case_of("gpt-oss", "decode", 1, 128, name="gpt-oss-decode-1"),
        # recurrent layers beside attention: many sequences
        case_of("redodra", "decode", 64, 512, name="redodra-decode-64"),
        # recurrent layers over long prompts
        case_of("redodra", "prefill", 4, 2048, name="redodra-prefill"),
        # the 32-bit option: one prompt of a trace replay
        case_of("redodra", "prefill", 1, 301, dtype="float32", name="redodra-prefill-fp32"),
    ]


def _spread(rng, lo, hi):
    """A whole number, uniform in the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    model = rng.choice(["llama", "llama", "llama", "qwen3", "qwen3", "gpt-oss", "redodra", "redodra"])
    mode = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed"])
    ragged = rng.random() < 0.5
    if model == "redodra" and rng.random() < 0.2:
        batch = rng.randint(1, 3)
        return case_of(model, "prefill", batch, _spread(rng, 16, 300 // batch), ragged, dtype="float32")
    if mode == "prefill":
        batch = _spread(rng, 1, 16)
        return case_of(model, mode, batch, _spread(rng, 16, min(8192, CHUNK // 2 // batch)), ragged)
    batch = _spread(rng, 1, 128)
    if mode == "mixed":
        batch = min(batch, 48)
    portion = _spread(rng, 16, 1024) if mode == "mixed" else 0
    return case_of(model, mode, batch, _spread(rng, 16, min(8000, 65536 // batch)), ragged, portion)


# --------------------------------------------------------------------------- inputs
def lengths(case):
    n = case["length"]
    if not case["ragged"]:
        return [n] * case["batch"]
    r = random.Random(n * 131 + case["batch"])
    return [n] + [r.randint((n + 1) // 2, n) for _ in range(case["batch"] - 1)]


class Draws:
    """Random tensors, each from the seed and its place in the order of creation."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=0.02, mean=0.0):
        x = torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(0.0, std, generator=self.g)
        return x + mean if mean else x


def ones(n):
    return torch.ones(n, dtype=torch.bfloat16, device=DEV)


def transformer_weights(cfg, d):
    """Hidden states of size 1 from the embedding on; a router that decides, as a trained one does."""
    H, V, D, E = cfg.hidden_size, cfg.vocab_size, cfg.head_dim, cfg.num_experts
    qkv, moe_i, ff = cfg.q_size + 2 * cfg.kv_size, cfg.moe_intermediate_size, cfg.intermediate_size
    w = {"tok_embedding": d.normal(V, H, std=1.0), "norm_weight": ones(H), "lm_head_weight": d.normal(H, V)}
    for i in range(cfg.num_layers):
        # YaRN multiplies scores by its concentration twice: smaller projections keep them of size one
        std = 0.02 if cfg.rope_scaling_factor <= 1 else 0.012
        t = {"qkv_weight": d.normal(H, qkv, std=std), "o_weight": d.normal(cfg.q_size, H),
             "input_layernorm_weight": ones(H), "post_attention_layernorm_weight": ones(H)}
        if cfg.qk_norm:
            t.update(q_norm_weight=ones(D), k_norm_weight=ones(D))
        if cfg.attn_bias:
            t.update(qkv_bias=d.normal(qkv), o_bias=d.normal(H))
        if cfg.attention_sinks:
            t["sinks"] = d.normal(cfg.num_heads, std=1.0).float()
        if E:
            t.update(router_weight=d.normal(H, E, std=0.1), gate_up_weight=d.normal(E, H, 2 * moe_i), down_weight=d.normal(E, moe_i, H))
            if cfg.router_bias:
                t["router_bias"] = d.normal(E)
            if cfg.expert_bias:
                t.update(gate_up_bias=d.normal(E, 2 * moe_i), down_bias=d.normal(E, H))
        else:
            t.update(gate_up_weight=d.normal(H, 2 * ff), down_weight=d.normal(ff, H))
        w.update({f"layers.{i}.{k}": v for k, v in t.items()})
    return w


def attention_tensors(m, W, d):
    rows = {"q": m.heads * m.dim, "k": m.kv_heads * m.dim, "v": m.kv_heads * m.vdim}
    t = {k: d.normal(n, W) for k, n in rows.items()}
    t["o"] = d.normal(W, m.heads * m.vdim)
    if m.bias:
        t.update({k + ".b": d.normal(n) for k, n in {**rows, "o": W}.items()})
    if m.distance:
        t.update(r1=ones(m.heads), r2=0.1 * ones(m.heads))
    if m.sink:
        t["sink"] = d.normal(m.heads)
    if m.gate:
        t["g"] = d.normal(m.heads, W)
    return t


def redodra_weights(cfg, d):
    """Decays of a memory of some fifty tokens, averages over the depth near their last term."""
    W, V = cfg.hidden_size, cfg.vocab_size

    def norm(name):
        return {name: ones(W), name + ".b": d.normal(W), name + ".alpha": ones(1)[0]}

    w = {"embed": d.normal(V, W, std=1.0), "head": d.normal(V, W), **norm("final.norm")}
    for i, layer in enumerate(cfg.layers):
        m = layer.mixer
        if m.kind == "delta":
            c, n = m.kv_heads * m.dim, m.heads * m.vdim
            mix = {"q": d.normal(c, W), "k": d.normal(c, W), "v": d.normal(n, W), "g": d.normal(n, W), "o": d.normal(W, n),
                   "b": d.normal(m.heads, W), "a": d.normal(m.heads, W), "norm": ones(m.vdim)}
            mix.update({x + ".conv": d.normal(len(mix[x]), m.conv, std=m.conv ** -0.5) for x in "qkv"})
            mix.update(A_log=d.normal(m.heads, mean=-2.0), dt_bias=d.normal(m.heads, mean=-2.0))
        elif m.kind == "blend":
            r = m.right
            n, ch = r.heads * r.vdim, r.heads * r.vdim + 2 * r.groups * r.state
            mix = {"left." + k: v for k, v in attention_tensors(m.left, W, d).items()}
            mix.update({"right.in": d.normal(n + ch + r.heads, W), "right.conv": d.normal(ch, r.conv, std=r.conv ** -0.5),
                        "right.conv.b": d.normal(ch), "right.dt_bias": d.normal(r.heads, mean=-2.0),
                        "right.A_log": d.normal(r.heads, mean=-2.0), "right.D": ones(r.heads), "right.norm": ones(n),
                        "right.o": d.normal(W, n), "left.out": ones(W), "right.out": ones(W)})
        else:
            mix = attention_tensors(m, W, d)
        t = {**norm("norm1"), **norm("norm1b"), **norm("norm2"), **norm("norm2b"), **{"mix." + k: v for k, v in mix.items()},
             "dwa": d.normal(i + 2), "mlp.up": d.normal(layer.ff, W), "mlp.down": d.normal(W, layer.ff), "mlp.act": d.normal(2)}
        t["dwa"][-1] += 1.0
        w.update({f"l{i}.{k}": v for k, v in t.items()})
    return w


def inputs(case, seed):
    """(configuration, weights, prompts, the token that follows each, the prompt that joins a mixed step)."""
    cfg, d = CONFIGS[case["model"]](), Draws(seed)
    w = redodra_weights(cfg, d) if cfg.layers else transformer_weights(cfg, d)
    g = torch.Generator().manual_seed(seed)
    ids = lambda n: torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist()
    return cfg, w, [ids(n) for n in lengths(case)], [ids(1) for _ in range(case["batch"])], ids(case["portion"])


class State:
    pass


def prepare(case, seed):
    s = State()
    cfg, w, s.prompts, s.follow, s.joins = inputs(case, seed)
    s.mode = case["mode"]
    model = registry.build(registry.for_config(cfg), cfg, w, None, DEV, getattr(torch, case["dtype"]))
    del w
    longest = max(max(map(len, s.prompts)) + 1, len(s.joins))
    # passes repeat the same prompts, which a shared prefix would turn into no work
    s.engine = eng = GenerationEngine(model, max_batch=case["batch"] + bool(s.joins), max_seq_len=longest + 31,
                                      prefill_chunk_tokens=CHUNK, enable_prefix_sharing=False)
    if s.mode != "prefill":
        s.open, step, room = [eng.open_request() for _ in s.prompts], [], CHUNK
        for seq, p in zip(s.open, s.prompts):
            if len(p) > room:
                eng.run_step(step)
                step, room = [], CHUNK
            step.append(StepEntry(seq, p))
            room -= len(p)
        eng.run_step(step)
        if s.mode == "decode":
            eng.prepare_decode(0, reserve=False)
    return s


def run(s):
    """One step of a scheduler; the logits behind the last token of every sequence."""
    eng = s.engine
    if s.mode == "prefill":
        seqs = [eng.open_request() for _ in s.prompts]
        logits = eng.run_step([StepEntry(q, p, [len(p) - 1]) for q, p in zip(seqs, s.prompts)])
        eng.release(seqs)
        return logits
    entries = [StepEntry(q, t, [0]) for q, t in zip(s.open, s.follow)]
    if s.mode == "mixed":
        new = eng.open_request()
        logits = eng.run_step(entries + [StepEntry(new, s.joins, [len(s.joins) - 1])])
        eng.release([new])
    else:
        logits = eng.run_step(entries)
    for q, p in zip(s.open, s.prompts):
        q.num_computed = len(p)          # the token is taken back, as a rejected draft is
    return logits


# --------------------------------------------------------------------------- what a pass needs
def work(case):
    """Every weight that a token meets and every visible key, value and state once, new ones and logits written."""
    cfg, lens = CONFIGS[case["model"]](), lengths(case)
    # (tokens before the new ones, new tokens) of every sequence
    spans = [(0, n) for n in lens] if case["mode"] == "prefill" else [(n, 1) for n in lens]
    if case["mode"] == "mixed":
        spans.append((0, case["portion"]))
    T, B, H, V = sum(n for _, n in spans), len(spans), cfg.hidden_size, cfg.vocab_size
    size = 4 if case["dtype"] == "float32" else 2
    seen = lambda p, n, w: sum(min(p + j + 1, w or p + j + 1) for j in range(n))
    flops, moved = 2.0 * B * V * H, H * V * size + 2 * T * H * size + B * V * (4 if cfg.layers else 2)

    def attention(heads, kv, dim, window=0):
        nonlocal flops, moved
        flops += 4.0 * heads * dim * sum(seen(p, n, window) for p, n in spans)
        moved += 2 * kv * dim * size * sum(min(p, window or p) + n for p, n in spans)

    def dense(n, tokens=T):
        nonlocal flops, moved
        flops += 2.0 * n * tokens
        moved += n * size

    for i in range(cfg.num_layers):
        if not cfg.layers:
            dense(H * (cfg.q_size + 2 * cfg.kv_size) + cfg.q_size * H)
            attention(cfg.num_heads, cfg.num_kv_heads, cfg.head_dim, cfg.window_for_layer(i))
            if not cfg.is_moe:
                dense(3 * H * cfg.intermediate_size)
                continue
            E, k, one = cfg.num_experts, cfg.top_k, 3 * H * cfg.moe_intermediate_size
            dense(H * E)
            flops += 2.0 * one * T * k
            moved += one * size * E * (1 - (1 - k / E) ** T)
            continue
        layer, m = cfg.layers[i], cfg.layers[i].mixer
        dense(2 * H * layer.ff)
        r = m if m.kind == "delta" else getattr(m, "right", None)
        a = m if m.kind == "grouped" else getattr(m, "left", None)
        if a is not None:
            dense(H * (2 * a.heads * a.dim + 2 * a.kv_heads * a.dim))
            attention(a.heads, a.kv_heads, a.dim, a.window)
        if r is not None:
            d = r.dim if m.kind == "delta" else r.state
            inner, rows = r.heads * r.vdim, 2 * (r.kv_heads if m.kind == "delta" else r.groups) * d
            dense(H * (3 * inner + rows))
            flops += 6.0 * r.heads * d * r.vdim * T
            moved += 8 * r.heads * d * r.vdim * B
    return {"bytes": float(moved), "flops": float(flops)}


def tolerance(case):
    # measured against `exact` and between two split-K factors: 1.2e-5 in 32 bits; bf16 0.006 to 0.014, single values 0.08
    if case["dtype"] == "float32":
        return {"rel": 5e-5, "max": 2e-3}
    return {"rel": 0.03, "max": 0.3}


# --------------------------------------------------------------------------- the same in 64 bits
def by_rows(f, x, n=8192):
    return torch.cat([f(p) for p in x.split(n)])


def rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def visible(n, window=0, keep=0):
    i = torch.arange(n, device=DEV)
    far = i[:, None] - i[None, :]
    return (far >= 0) & ((far < (window or n)) | (i[None, :] < keep)), far


def attend(q, k, v, scale, window=0, keep=0, sink=None, cap=0.0, dist=None):
    """q [n, heads, dim], k and v [n, kv heads, dim] of one sequence."""
    n, heads, dim = q.shape
    mask, far = visible(n, window, keep)
    out, group = torch.empty_like(q), heads // k.shape[1]
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T).mul_(scale)
        if cap:
            s = cap * torch.tanh(s / cap)
        if dist is not None:
            s -= dist[0][h] * torch.log1p(dist[1][h] * far.clamp(min=0).double())
        s.masked_fill_(~mask, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[h])
        s = s.sub_(top).exp_()
        total = s.sum(-1, keepdim=True)
        if sink is not None:
            total += torch.exp(sink[h] - top)
        out[:, h] = (s @ v[:, h // group]) / total
    return out.reshape(n, -1)


def each(f, lens, *xs):
    """f on the rows of every sequence."""
    return torch.cat([f(*p) for p in zip(*(x.split(lens) for x in xs))])


def transformer_exact(cfg, w, seqs):
    lens, D, nq, nkv = [len(s) for s in seqs], cfg.head_dim, cfg.num_heads, cfg.num_kv_heads
    W = lambda name: w[name].double()
    x = W("tok_embedding")[torch.tensor(sum(seqs, []), device=DEV)]
    freq, mult = rotations(cfg)
    at = torch.cat([torch.arange(n, device=DEV) for n in lens]).double()[:, None] * freq
    cos, sin = (at.cos() * mult)[:, None], (at.sin() * mult)[:, None]

    def rope(t):
        a, b = t.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def act(h):
        g, u = h.chunk(2, -1)
        if cfg.swiglu_limit > 0:
            g, u = g.clamp(max=cfg.swiglu_limit), u.clamp(-cfg.swiglu_limit, cfg.swiglu_limit) + 1
            return u * g * torch.sigmoid(cfg.swiglu_alpha * g)
        return F.silu(g) * u

    for i in range(cfg.num_layers):
        p = f"layers.{i}."
        b = lambda name, on: W(p + name) if on else 0.0
        wt = W(p + "qkv_weight")
        qkv = by_rows(lambda r: rms(r, cfg.rms_eps) @ wt, x) + b("qkv_bias", cfg.attn_bias)
        q, k, v = (t.view(len(x), -1, D) for t in qkv.split([nq * D, nkv * D, nkv * D], -1))
        if cfg.qk_norm:
            q, k = rms(q, cfg.rms_eps), rms(k, cfg.rms_eps)
        sink = W(p + "sinks") if cfg.attention_sinks else None
        o = each(lambda *t: attend(*t, D ** -0.5, cfg.window_for_layer(i), sink=sink), lens, rope(q), rope(k), v)
        x = x + o @ W(p + "o_weight") + b("o_bias", cfg.attn_bias)
        h = rms(x, cfg.rms_eps)
        if not cfg.is_moe:
            up, down = W(p + "gate_up_weight"), W(p + "down_weight")
            x = x + by_rows(lambda r: act(r @ up) @ down, h)
            continue
        z = h @ W(p + "router_weight") + b("router_bias", cfg.router_bias)
        if cfg.router_mode == "softmax_topk":
            share, pick = torch.softmax(z, -1).topk(cfg.top_k, -1)
            share = share / share.sum(-1, keepdim=True)
        else:
            share, pick = z.topk(cfg.top_k, -1)
            share = torch.softmax(share, -1)
        for e in range(cfg.num_experts):
            rows, place = (pick == e).nonzero(as_tuple=True)
            bias = (w[p + "gate_up_bias"][e].double(), w[p + "down_bias"][e].double()) if cfg.expert_bias else (0.0, 0.0)
            y = act(h[rows] @ w[p + "gate_up_weight"][e].double() + bias[0]) @ w[p + "down_weight"][e].double() + bias[1]
            x.index_add_(0, rows, y * share[rows, place][:, None])
    last = torch.tensor(lens, device=DEV).cumsum(0) - 1
    return rms(x[last], cfg.rms_eps) @ W("lm_head_weight")


def rotations(cfg):
    """Frequencies of the rotary embedding and the multiplier of its cosines and sines (YaRN with a factor)."""
    D, base, f = cfg.head_dim, cfg.rope_theta, cfg.rope_scaling_factor
    j = torch.arange(D // 2, dtype=torch.float64, device=DEV)
    plain = base ** (-2 * j / D)
    if f <= 1:
        return plain, 1.0
    bound = lambda turns: D / 2 * math.log(cfg.rope_original_max_position / (turns * 2 * math.pi)) / math.log(base)
    low, high = bound(cfg.rope_beta_fast), bound(cfg.rope_beta_slow)
    keep = 1 - ((j - low) / (high - low)).clamp(0, 1)
    return plain * keep + plain / f * (1 - keep), 0.1 * math.log(f) + 1.0


def padded(x, lens):
    """[tokens, ...] -> [sequences, longest, ...], zeros behind the end."""
    return torch.nn.utils.rnn.pad_sequence(x.split(lens), batch_first=True)


def packed(x, lens):
    return torch.cat([x[i, :n] for i, n in enumerate(lens)])


def short_conv(x, taps, bias, lens):
    """x [tokens, channels], taps [channels, n], the last column for the current token."""
    def one(p):
        q = F.pad(p, (0, 0, taps.shape[1] - 1, 0))
        return sum(q[i:i + len(p)] * taps[:, i] for i in range(taps.shape[1]))

    return F.silu(each(one, lens, x) + bias)


def scan(q, k, write, decay, lens):
    """S <- decay S, S <- S + k write(t, S)^T, out = S^T q; q, k [tokens, heads, dim], decay [tokens, heads]."""
    q, k, decay = padded(q, lens), padded(k, lens), padded(decay, lens)
    state, outs = None, []
    for t in range(q.shape[1]):
        if state is None:
            state = q.new_zeros((*k[:, t].shape, write(0, None).shape[-1]))
        state = state * decay[:, t, :, None, None]
        state = state + k[:, t, :, :, None] * write(t, state)[:, :, None, :]
        outs.append(torch.einsum("bhdn,bhd->bhn", state, q[:, t]))
    return packed(torch.stack(outs, 1), lens)


def redodra_exact(cfg, w, seqs):
    lens, eps = [len(s) for s in seqs], cfg.rms_eps
    N = sum(lens)
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).double()
    W = lambda name: w[name].double()
    norm = lambda x, name: torch.tanh(W(name + ".alpha") * x) * W(name) + W(name + ".b")
    unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)

    def rope(t, spec):
        i = torch.arange(spec.dims // 2, device=DEV).double()
        at = (pos[:, None] * spec.base ** (-2 * i / spec.dims))[:, None]
        u, v = t[..., 0:spec.dims:2], t[..., 1:spec.dims:2]
        turned = torch.stack([u * at.cos() - v * at.sin(), v * at.cos() + u * at.sin()], -1).flatten(-2)
        return torch.cat([turned, t[..., spec.dims:]], -1)

    def attention(h, m, p):
        b = lambda n: W(p + n + ".b") if m.bias else 0.0
        q, k, v = ((h @ W(p + n).T + b(n)).view(N, -1, m.dim) for n in "qkv")
        if m.rope:
            q, k = rope(q, m.rope), rope(k, m.rope)
        o = each(lambda *t: attend(*t, m.scale, m.window, m.keep_first if m.window else 0, W(p + "sink") if m.sink else None,
                                   m.softcap, (W(p + "r1"), W(p + "r2")) if m.distance else None), lens, q, k, v)
        if m.gate:
            o = (o.view(N, m.heads, -1) * torch.sigmoid(h @ W(p + "g").T)[..., None]).flatten(1)
        return o @ W(p + "o").T + b("o")

    def delta(h, m, p):
        q, k, v = (short_conv(h @ W(p + n).T, W(p + n + ".conv"), 0.0, lens).view(N, -1, m.dim) for n in "qkv")
        q, k = (t.repeat_interleave(m.heads // m.kv_heads, 1) for t in (unit(q) * m.dim ** -0.5, unit(k)))
        beta = padded(torch.sigmoid(h @ W(p + "b").T), lens)
        decay = torch.exp(-torch.exp(W(p + "A_log")) * F.softplus(h @ W(p + "a").T + W(p + "dt_bias"), threshold=200.0))
        ks, vs = padded(k, lens), padded(v, lens)
        write = lambda t, S: (beta[:, t, :, None] * (vs[:, t] - torch.einsum("bhdn,bhd->bhn", S, ks[:, t]))
                              if S is not None else vs[:, t])
        o = rms(scan(q, k, write, decay, lens), eps) * W(p + "norm")
        return (o.flatten(1) * F.silu(h @ W(p + "g").T)) @ W(p + "o").T

    def state_space(h, m, p):
        n, c = m.heads * m.vdim, m.groups * m.state
        z, xbc, dt = (h @ W(p + "in").T).split([n, n + 2 * c, m.heads], -1)
        x, B, Cq = short_conv(xbc, W(p + "conv"), W(p + "conv.b"), lens).split([n, c, c], -1)
        x = x.reshape(N, m.heads, m.vdim)
        B, Cq = (t.reshape(N, m.groups, m.state).repeat_interleave(m.heads // m.groups, 1) for t in (B, Cq))
        dt = F.softplus(dt + W(p + "dt_bias"), threshold=200.0)
        xs = padded(x * dt[..., None], lens)
        y = scan(Cq, B, lambda t, S: xs[:, t], torch.exp(-torch.exp(W(p + "A_log")) * dt), lens)
        y = (y + W(p + "D")[:, None] * x).flatten(1) * F.silu(z)
        return (rms(y.view(N, m.norm_groups, -1), eps).flatten(1) * W(p + "norm")) @ W(p + "o").T

    x = W("embed")[torch.tensor(sum(seqs, []), device=DEV)]
    results = [x]
    for i, layer in enumerate(cfg.layers):
        p, m = f"l{i}.", layer.mixer
        h, mix = norm(x, p + "norm1"), p + "mix."
        if m.kind == "delta":
            y = delta(h, m, mix)
        elif m.kind == "blend":
            y = (rms(attention(h, m.left, mix + "left."), eps) * W(mix + "left.out")
                 + rms(state_space(h, m.right, mix + "right."), eps) * W(mix + "right.out")) / 2
        else:
            y = attention(h, m, mix)
        x = x + norm(y, p + "norm1b")
        pos_a, neg_a = F.softplus(W(p + "mlp.act"), threshold=200.0).tolist()
        up, down = W(p + "mlp.up"), W(p + "mlp.down")

        def mlp(r):
            z = r @ up.T
            return torch.where(z > 0, pos_a * z * z, (0.5 + neg_a) * (torch.expm1(z) - z)).add_(z / 2) @ down.T

        x = x + norm(by_rows(mlp, norm(x, p + "norm2")), p + "norm2b")
        results.append(x)
        x = sum(a * r for a, r in zip(W(p + "dwa"), results))
    last = torch.tensor(lens, device=DEV).cumsum(0) - 1
    return norm(x[last], "final.norm") @ W("head").T


def exact(case, seed):
    whole = sum(lengths(case)) + case["portion"]
    cfg = CONFIGS[case["model"]]()
    if whole * cfg.param_count() * (cfg.top_k / cfg.num_experts if cfg.is_moe else 1) > 2e14:
        return None                      # too long in 64 bits
    cfg, w, prompts, follow, joins = inputs(case, seed)
    if case["mode"] != "prefill":
        prompts = [p + t for p, t in zip(prompts, follow)]
    seqs = prompts + ([joins] if joins else [])
    with torch.no_grad():
        return redodra_exact(cfg, w, seqs) if cfg.layers else transformer_exact(cfg, w, seqs)
