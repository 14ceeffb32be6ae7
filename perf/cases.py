"""Measured cases: rounds of the token loop through the public binding (`Context.step`), with weights of the shapes in
`llama_cu_b200.CONFIGS`.

A case is one pass of one of these kinds:

  decode    one round that brings one token per sequence; the sequences' prompts are in the cache already
  prefill   one round that brings a whole prompt of a new sequence
  mixed     one round of continuous batching: a token of every running sequence and the last part of a new prompt that came
            in parts; every second request is sampled with temperature, top-k and top-p
  request   a layered model from prompt to answer: one round with the prompts of all sequences, then rounds of one token each

Tokens come from the host, as in a service that streams its answers.  A pass returns the logits of every request and (models
of the LLaMA family) the residual stream after the last layer, rounds with running sequences also the cache they appended to.
Sampled tokens stay out: they follow from the logits, and a tie between the two largest of random logits is no error.
"""
import functools
import math
from dataclasses import replace

import numpy as np
import torch

import llama_cu_b200 as L
from llama_cu_b200 import galarax, layered

DEV = "cuda:0"

# the settings of `lcu_sample_args` that a chat service uses
SAMPLING = (0.8, 0.95, 50)


def listed():
    return [
        # the smallest call: two layers, one sequence; launches and host work are all there is
        {"name": "decode-tiny-f16-b1", "kind": "decode", "model": "tiny", "layers": 2, "batch": 1, "short": 16, "long": 16},
        # one user, small model: short kernels in a row
        {"name": "decode-1b-bf16-b1", "kind": "decode", "model": "llama1b", "layers": 16, "batch": 1, "short": 199, "long": 199},
        # one user, the benchmark's own workload: weights stream once per token
        {"name": "decode-8b-f16-b1", "kind": "decode", "model": "llama8b", "layers": 32, "batch": 1, "short": 128, "long": 128},
        # a service under load: 32 conversations of uneven length
        {"name": "decode-8b-f16-b32", "kind": "decode", "model": "llama8b", "layers": 32, "batch": 32, "short": 128, "long": 1024},
        # the same two with quantised weights
        {"name": "decode-8b-q8-b1", "kind": "decode", "model": "llama8b_q8", "layers": 32, "batch": 1, "short": 128, "long": 128},
        {"name": "decode-8b-q8-b16", "kind": "decode", "model": "llama8b_q8", "layers": 32, "batch": 16, "short": 100, "long": 290},
        # a short chat message
        {"name": "prefill-1b-bf16-33", "kind": "prefill", "model": "llama1b", "layers": 16, "tokens": 33},
        # a page of text, just below the reference's limit of a round
        {"name": "prefill-8b-f16-997", "kind": "prefill", "model": "llama8b", "layers": 32, "tokens": 997},
        {"name": "prefill-8b-q8-500", "kind": "prefill", "model": "llama8b_q8", "layers": 32, "tokens": 500},
        # a long document: attention weighs as much as the matrices
        {"name": "prefill-1b-bf16-8000", "kind": "prefill", "model": "llama1b", "layers": 16, "tokens": 8000},
        # continuous batching with a prompt that arrives in parts
        {"name": "mixed-8b-f16-b31", "kind": "mixed", "model": "llama8b", "layers": 32, "batch": 31, "short": 60, "long": 700, "past": 512, "tokens": 481},
        # a layered model (softmax attention beside a gated delta rule), prompt and first words of the answer
        {"name": "request-galarax8b-2000", "kind": "request", "model": "galarax8b", "layers": 8, "vocab": 32000, "batch": 1, "tokens": 2000, "rounds": 8},
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Models of the listed kinds and types with fewer layers (all layers of a model are alike), any batch up to the largest
    round of 64 requests, any length."""
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed", "request"])
    if kind == "request":
        model = rng.choice(["galarax8b", "galarax1b"])
        batch = log_uniform(rng, 1, 12)
        return {"kind": kind, "model": model, "layers": rng.randint(2, 4), "vocab": 32000, "batch": batch,
                "tokens": log_uniform(rng, 5, 2000 // batch), "rounds": rng.randint(1, 6)}
    model = rng.choice(["tiny", "llama1b", "llama8b", "llama8b_q8"])
    case = {"kind": kind, "model": model, "layers": {"tiny": 2, "llama1b": rng.randint(4, 16)}.get(model, rng.randint(2, 8))}
    most = L.CONFIGS[model].nctx - 64
    if kind != "prefill":
        case["batch"] = log_uniform(rng, 1, 64 if kind == "decode" else 48)
        case["short"] = log_uniform(rng, 1, most)
        case["long"] = min(most, case["short"] + rng.randint(0, 400))
    if kind != "decode":
        case["past"] = log_uniform(rng, 16, most // 2) if kind == "mixed" else 0
        case["tokens"] = log_uniform(rng, 3, most // 2 if kind == "mixed" else most)
    return case


# ---------------------------------------------------------------------------------------------------------------------- inputs

def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def llama_config(case):
    cfg = L.CONFIGS[case["model"]]
    return replace(cfg, n_layers=case["layers"], nctx=max(cfg.nctx, case.get("tokens", 0) + 64))


def llama_weights(case, seed):
    """Yields ((layer, kind), tensor): normal matrices, norms around one; Q8_0 as a pair (int8 values, f16 scales)."""
    cfg, g = llama_config(case), generator(seed)
    dt = L.torch_dtype(cfg.act_dtype)

    def normal(*shape, std=0.02, mean=0.0):
        return torch.empty(shape, dtype=dt, device=DEV).normal_(mean, std, generator=g)

    def matrix(rows, cols):
        if cfg.wdt != L.Q8_0:
            return normal(rows, cols)
        q = torch.randint(-127, 128, (rows, cols), dtype=torch.int8, device=DEV, generator=g)
        return q, torch.empty(rows, cols // 32, device=DEV).uniform_(1e-4, 4e-4, generator=g).half()

    sh = cfg.shapes()
    yield (0, L.W_EMBD), normal(*sh[L.W_EMBD])
    for i in range(cfg.n_layers):
        for kind in (L.W_ATTN_NORM, L.W_QKV, L.W_O, L.W_FFN_NORM, L.W_GATE_UP, L.W_DOWN):
            yield (i, kind), matrix(*sh[kind]) if kind in L.LINEAR_KINDS else normal(*sh[kind], std=0.1, mean=1.0)
    yield (0, L.W_OUT_NORM), normal(*sh[L.W_OUT_NORM], std=0.1, mean=1.0)
    yield (0, L.W_LM_HEAD), normal(*sh[L.W_LM_HEAD])


def galarax_config(case):
    cfg = L.CONFIGS[case["model"]]
    return replace(cfg, layers=cfg.layers[:case["layers"]], vocab=case["vocab"], act_dtype=L.BF16)


def galarax_tensors(case, seed):
    """{name: bf16 tensor} as a model file would hold them."""
    g, out = generator(seed), {}
    for name, shape in galarax.tensor_shapes(galarax_config(case)).items():
        w, last = torch.randn(shape, generator=g, device=DEV), name.rsplit(".", 1)[-1]
        if name.endswith("right.norm") or last == "out":
            w = 1 + 0.1 * w
        elif last in ("norm1", "norm2", "norm") or last == "b" and len(shape) == 1:
            w = 0.2 * w
        elif last in ("A_log", "dt_bias"):
            w = w - 1.2
        elif name != "embed":
            w = w / shape[-1] ** 0.5
        out[name] = w.bfloat16()
    return out


def lengths(case):
    """Tokens that each running sequence holds: spread evenly from the shortest to the longest, in no order."""
    n = case.get("batch", 0)
    if "short" not in case:
        return []
    return [case["short"] + (case["long"] - case["short"]) * ((i * 13) % n) // max(n - 1, 1) for i in range(n)]


def prompts(case, seed):
    """Token ids of every sequence up to and with the measured round, running sequences first."""
    vocab = case.get("vocab", L.CONFIGS[case["model"]].vocab)
    if case["kind"] == "request":
        sizes = [case["tokens"] + case["rounds"]] * case["batch"]
    else:
        sizes = [n + 1 for n in lengths(case)]
        if case["kind"] != "decode":
            sizes.append(case["past"] + case["tokens"] if case["kind"] == "mixed" else case["tokens"])
    rng = np.random.default_rng(seed)
    return [rng.integers(3, vocab, n).astype(np.uint32) for n in sizes]


class Device:
    """Device memory of a context, for torch.as_tensor; tensors made from it keep the context alive."""

    def __init__(self, ctx, address, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (address, False), "version": 2}


def view(ctx, address, rows, cols, dt):
    t = torch.as_tensor(Device(ctx, address, (rows, cols), "<f4" if dt == L.F32 else "<i2"), device=DEV)
    return t.view(L.torch_dtype(dt))


@functools.cache
def main_stream():
    """The one stream of the program: rounds of one token per request are captured, which stream 0 cannot be."""
    return torch.cuda.Stream(device=DEV)


def prepare(case, seed):
    """The loaded model, its cache, and the round to run."""
    toks = prompts(case, seed)
    kind = case["kind"]
    if kind == "request":
        cfg = galarax_config(case)
        ctx = L.Context(cfg.desc(max_tokens=max(1, case["batch"] * case["tokens"]), max_seqs=max(4, case["batch"])), 0, layers=cfg.layer_descs())
        weights = galarax.pack(cfg, layered.Tensors(galarax_tensors(case, seed)))
    else:
        cfg = llama_config(case)
        ctx = L.Context(cfg.desc(max_tokens=max(1024, sum(map(len, toks)) if kind == "prefill" else 0), max_seqs=max(4, len(toks))), 0)
        weights = llama_weights(case, seed)
    for (layer, k), w in weights:
        if isinstance(w, tuple):  # the library's layout of Q8_0: all values, then all scales
            w = torch.cat([w[0].view(torch.uint8).reshape(-1), w[1].view(torch.uint8).reshape(-1)])
        ctx.set_weight(max(layer, 0), k, w)
    del weights
    pages = sum(-(-len(t) // ctx.page_tokens) for t in toks)
    pool = torch.zeros(pages * ctx.page_bytes // 2, dtype=L.torch_dtype(cfg.act_dtype), device=DEV)
    ctx.kv_pool_attach(pool)
    seqs = [ctx.seq_create() for _ in toks]
    out = torch.zeros(len(toks), 2, dtype=torch.int32, device=DEV)
    stream = main_stream()
    stream.wait_stream(torch.cuda.current_stream())
    s = {"ctx": ctx, "out": out, "stream": stream, "rounds": [], "args": None, "randoms": None, "pool": pool if kind in ("decode", "mixed") else None}
    if kind == "request":
        n = case["tokens"]
        s["rounds"].append(([(q, 0, n) for q in seqs], np.concatenate([t[:n] for t in toks])))
        for r in range(case["rounds"]):
            s["rounds"].append(([(q, n + r, 1) for q in seqs], np.array([t[n + r] for t in toks])))
    else:
        new = [1] * len(toks)
        if kind != "decode":
            new[-1] = case["tokens"]
        for q, t, n in zip(seqs, toks, new):  # what came before the measured round
            for p in range(0, len(t) - n, 1024):
                part = t[p:min(p + 1024, len(t) - n)]
                ctx.step([(q, p, len(part))], part, out, stream=stream)
        s["rounds"].append(([(q, len(t) - n, n) for q, t, n in zip(seqs, toks, new)], np.concatenate([t[len(t) - n:] for t, n in zip(toks, new)])))
        if kind == "mixed":
            s["args"] = [L.SampleArgs.new(*SAMPLING) if i % 2 else L.SampleArgs.arg_max() for i in range(len(toks))]
            s["randoms"] = np.random.default_rng(seed + 1).random(len(toks), dtype=np.float32)
    stride = ctx.lib.lcu_logits_stride(ctx.h)
    s["logits"] = view(ctx, ctx.lib.lcu_logits(ctx.h), len(toks), stride, cfg.act_dtype)[:, :cfg.vocab]
    if kind != "request":
        s["hidden"] = view(ctx, ctx.lib.lcu_hidden(ctx.h), sum(n for _, _, n in s["rounds"][-1][0]), cfg.d, cfg.act_dtype)
    return s


def run(s):
    for reqs, tokens in s["rounds"]:
        s["ctx"].step(reqs, tokens, s["out"], args=s["args"], randoms=s["randoms"], stream=s["stream"])
    out = {"logits": s["logits"], "hidden": s.get("hidden"), "cache": s["pool"]}
    return {k: v for k, v in out.items() if v is not None}


# ------------------------------------------------------------------------------------------------------------------------ work

def work(case):
    """Every weight of a round read once, the cache of every request read once, logits written once; two operations per weight
    and token, four per query head, dimension and pair of tokens."""
    if case["kind"] == "request":
        cfg, rounds = galarax_config(case), 1 + case["rounds"]
        layer = sum(math.prod(s) for n, s in galarax.tensor_shapes(replace(cfg, layers=cfg.layers[:1])).items() if n.startswith("l0."))
        m, r = cfg.layers[0].mixer.left, cfg.layers[0].mixer.right
        n, seqs = case["tokens"], case["batch"]
        total = seqs * (n + case["rounds"])
        cache = cfg.n_layers * 2 * m.kv_heads * m.dim * 2
        state = cfg.n_layers * r.heads * r.dim * r.v_dim * 4
        head = cfg.vocab * cfg.d
        nbytes = rounds * (layer * cfg.n_layers + head) * 2 + seqs * (cache * n * rounds + state * 2 * rounds)
        pairs = seqs * (n + case["rounds"]) ** 2 / 2
        flops = 2.0 * total * layer * cfg.n_layers + 2.0 * seqs * rounds * head + cfg.n_layers * (
            4.0 * pairs * m.heads * m.dim + 8.0 * total * r.heads * r.dim * r.v_dim)
        return {"bytes": float(nbytes), "flops": flops}
    cfg = llama_config(case)
    new = [1] * len(lengths(case)) + ([case["tokens"]] if case["kind"] != "decode" else [])
    old = lengths(case) + ([case["past"] if case["kind"] == "mixed" else 0] if case["kind"] != "decode" else [])
    params = cfg.n_layers * sum(math.prod(cfg.shapes()[k]) for k in L.LINEAR_KINDS)
    head = cfg.vocab * cfg.d
    pairs = sum(n * o + n * (n + 1) / 2 for n, o in zip(new, old))
    nbytes = cfg.weight_bytes_per_step() + cfg.kv_bytes_per_token() * sum(n + o for n, o in zip(new, old)) + 2.0 * len(new) * cfg.vocab
    return {"bytes": nbytes, "flops": 2.0 * sum(new) * params + 2.0 * len(new) * head + 4.0 * cfg.n_layers * pairs * cfg.nh * cfg.dh}


def tolerance(case):
    """About four times what the library differs from the 64-bit result by: activations are rounded to 16 bits between
    operators, and every layer multiplies the error (measured: tiny 7e-4, 32 layers in f16 7e-3, 16 layers in bf16 2.5e-2, where
    the bound is just above; Galarax 5e-3)."""
    return {"rel": 0.003 if case["model"] == "tiny" else 0.02 if case["kind"] == "request" else 0.03}


# ---------------------------------------------------------------------------------------------------------------- in 64 bits

def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def attention(q, k, v, scale):
    """Causal, [tokens, heads, dim]; query head h reads key head h // (heads / kv_heads)."""
    n, group = q.shape[0], q.shape[1] // k.shape[1]
    mask = torch.ones(n, n, dtype=torch.bool, device=q.device).tril()
    out = torch.empty(n, q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T) * scale
        out[:, h] = torch.softmax(s.masked_fill_(~mask, -math.inf), -1) @ v[:, h // group]
    return out.reshape(n, -1)


def llama_exact(case, seed):
    cfg = llama_config(case)
    toks = prompts(case, seed)
    ends = np.cumsum([len(t) for t in toks])
    parts = [slice(e - len(t), e) for t, e in zip(toks, ends)]
    pos = torch.cat([torch.arange(len(t), device=DEV) for t in toks]).double()
    angle = pos[:, None] * cfg.theta ** (-torch.arange(0, cfg.dh, 2, device=DEV).double() / cfg.dh)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def rotate(x):  # neighbouring dimensions are a pair
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)

    def full(w):
        if isinstance(w, tuple):
            return (w[0].double().view(w[0].shape[0], -1, 32) * w[1].double()[..., None]).view(w[0].shape)
        return w.double()

    qd, kvd = cfg.nh * cfg.dh, cfg.nkvh * cfg.dh
    for (_, kind), w in llama_weights(case, seed):
        if kind == L.W_EMBD:
            x = w[torch.from_numpy(np.concatenate(toks).astype(np.int64)).to(DEV)].double()
        elif kind in (L.W_ATTN_NORM, L.W_FFN_NORM, L.W_OUT_NORM):
            if kind == L.W_OUT_NORM:
                x = torch.cat([x[p] for p in parts])
                new = [1] * len(toks)
                if case["kind"] != "decode":
                    new[-1] = case["tokens"]
                hidden = torch.cat([x[e - n:e] for e, n in zip(ends, new)])
                x = x[torch.from_numpy(ends - 1).to(DEV)]
            h = rms(x, cfg.eps) * w.double()
        elif kind == L.W_QKV:
            q, k, v = (h @ full(w).T).split([qd, kvd, kvd], 1)
            q, k, v = rotate(q.view(-1, cfg.nh, cfg.dh)), rotate(k.view(-1, cfg.nkvh, cfg.dh)), v.view(-1, cfg.nkvh, cfg.dh)
            h = torch.cat([attention(q[p], k[p], v[p], cfg.dh ** -0.5) for p in parts])
            del q, k, v
        elif kind == L.W_GATE_UP:
            g, u = (h @ full(w).T).chunk(2, 1)
            h = torch.nn.functional.silu(g).mul_(u)
            del g, u
        elif kind == L.W_LM_HEAD:
            return {"logits": h @ full(w).T, "hidden": hidden, "cache": None}
        else:
            x = x + h @ full(w).T


def yarn(rot):
    """(frequencies, factor on cos and sin)."""
    n = rot.dims
    freq = rot.base ** (-2.0 * torch.arange(n // 2, device=DEV).double() / n)

    def index_of(turns):
        return n * math.log(rot.original / (turns * 2 * math.pi)) / (2 * math.log(rot.base))
    lo, hi = max(math.floor(index_of(rot.fast)), 0), min(math.ceil(index_of(rot.slow)), n - 1)
    ramp = ((torch.arange(n // 2, device=DEV).double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return freq / rot.factor * ramp + freq * (1 - ramp), 0.1 * math.log(rot.factor) + 1


def conv(x, w):
    taps = w.shape[1]
    x = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(x[j:x.shape[0] - (taps - 1 - j)] * w[:, j] for j in range(taps))


def galarax_attention(h, w, m, eps):
    n, half = h.shape[0], m.rot.dims // 2
    freq, gain = yarn(m.rot)
    angle = torch.arange(n, device=DEV).double()[:, None] * freq
    cos, sin = (torch.cos(angle) * gain)[:, None], (torch.sin(angle) * gain)[:, None]

    def turn(x):
        a, b = x[..., :half], x[..., half:2 * half]
        return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., 2 * half:]], -1)
    q, k, v = (h @ w("left." + t).T + w("left." + t + ".b") for t in "qkv")
    q, k = rms(turn(q.view(n, m.heads, m.dim)), eps), rms(turn(k.view(n, m.kv_heads, m.dim)), eps)
    return attention(q, k, v.view(n, m.kv_heads, m.v_dim), m.scale) @ w("left.o").T


def galarax_delta(h, w, m, eps):
    n, silu = h.shape[0], torch.nn.functional.silu
    q, k, v = (silu(conv(h @ w("right." + t).T, w("right." + t + ".conv"))) for t in "qkv")
    q, k = (x.view(n, m.kv_heads, m.dim) for x in (q, k))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (x.repeat_interleave(m.heads // m.kv_heads, 1) for x in (q * m.dim ** -0.5, k))
    v = v.view(n, m.heads, m.v_dim)
    decay = torch.exp(-torch.exp(w("right.A_log")) * torch.nn.functional.softplus(h @ w("right.a").T + w("right.dt_bias")))
    beta = torch.sigmoid(h @ w("right.b").T)
    s, out = h.new_zeros(m.heads, m.dim, m.v_dim), []
    for t in range(n):  # the state decays, is corrected towards v along k, then read along q
        s = s * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], s)[:, 0])
        s = torch.baddbmm(s, k[t, :, :, None], u[:, None])
        out.append(torch.bmm(q[t, :, None], s)[:, 0])
    o = rms(torch.stack(out), eps) * w("right.norm") * silu(h @ w("right.g").T).view(n, m.heads, m.v_dim)
    return o.reshape(n, -1) @ w("right.o").T


def galarax_exact(case, seed):
    cfg, t = galarax_config(case), galarax_tensors(case, seed)
    logits = []
    for ids in prompts(case, seed):
        x = t["embed"][torch.from_numpy(ids.astype(np.int64)).to(DEV)].double()
        for i, l in enumerate(cfg.layers):
            h = rms(x, cfg.eps) * (1 + t[f"l{i}.norm1"].double())

            def w(name):
                return t[f"l{i}.mix." + name].double()
            x = x + (rms(galarax_attention(h, w, l.mixer.left, cfg.eps), cfg.eps) * w("left.out")
                     + rms(galarax_delta(h, w, l.mixer.right, cfg.eps), cfg.eps) * w("right.out")) / 2
            h = rms(x, cfg.eps) * (1 + t[f"l{i}.norm2"].double())
            x = x + torch.relu(h @ t[f"l{i}.mlp.up"].double().T).square() @ t[f"l{i}.mlp.down"].double().T
        logits.append((rms(x[-1], cfg.eps) * (1 + t["final.norm"].double())) @ t["head"].double().T)
    return {"logits": torch.stack(logits)}


def exact(case, seed):
    with torch.no_grad():
        return galarax_exact(case, seed) if case["kind"] == "request" else llama_exact(case, seed)
