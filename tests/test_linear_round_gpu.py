"""Linear layers inside a round, where they own scratch: row blocks cut between CTAs and merged, clusters beside them, against f64
products of one projection; and the epilogues of layered models on the 256-row tiles.

A model of one layer whose value rows copy the normed input (one weight of 1 a row) and whose down projection is zero: sequences at
their first token attend to themselves alone, so the input of the output projection is known exactly, and the residual stream after the
layer is its result."""
import importlib
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def default_tuning(L):
    yield
    for k, v in (("tc", 1), ("tc_cluster", 1), ("tc_pair_min", 129)):
        L.set_tuning(k, v)


def plane(L, q8, w, gen):
    """A matrix as the library holds it, and in f64."""
    if not q8:
        return w, w.double()
    rows, cols = w.shape
    s = torch.empty(rows, cols // 32, device=DEV).uniform_(1e-4, 4e-4, generator=gen).half()
    q = torch.randint(-128, 128, (rows, cols), dtype=torch.int8, device=DEV, generator=gen)
    return torch.cat([q.view(torch.uint8).reshape(-1), s.view(torch.uint8).reshape(-1)]), (q.double().view(rows, -1, 32) * s.double()[..., None]).view(rows, cols)


def one_per_row(L, q8, at, cols, dt):
    """Row i holds 1 in column at[i]."""
    rows = len(at)
    if not q8:
        w = torch.zeros(rows, cols, device=DEV, dtype=dt)
        w[torch.arange(rows), at] = 1
        return w
    q = torch.zeros(rows, cols, dtype=torch.int8, device=DEV)
    q[torch.arange(rows), at] = 1
    return torch.cat([q.view(torch.uint8).reshape(-1), torch.ones(rows, cols // 32, device=DEV, dtype=torch.float16).view(torch.uint8).reshape(-1)])


def one_layer(L, act, q8, d, nh, di, n, what, embd=None):
    """The context and the f64 matrix of `what` ("o": the output projection, "ffn": gates and ups)."""
    dt = L.torch_dtype(act)
    cfg = replace(L.CONFIGS["tiny"], n_layers=1, d=d, nh=nh, nkvh=nh, dh=128, di=di, vocab=512, act_dtype=act, weight_dtype=L.Q8_0 if q8 else -1, nctx=128)
    g = torch.Generator(device=DEV)
    g.manual_seed(d + nh + n)
    ctx = L.Context(cfg.desc(max_tokens=128, max_seqs=128), 0)
    k = nh * 128
    zero = (lambda r, c: torch.zeros(r * c + r * c // 16, dtype=torch.uint8, device=DEV)) if q8 else (lambda r, c: torch.zeros(r, c, device=DEV, dtype=dt))
    normal = lambda r, c: torch.randn(r, c, device=DEV, generator=g).mul_(0.05).to(dt)
    at = (torch.arange(k, device=DEV) % d).repeat(3)
    qkv = one_per_row(L, q8, at, d, dt)
    embd = torch.randn(cfg.vocab, d, device=DEV, generator=g).to(dt) if embd is None else embd(cfg, g, dt)
    o, o64 = plane(L, q8, normal(d, k), g) if what == "o" else (zero(d, k), None)
    gu, gu64 = plane(L, q8, normal(2 * di, d), g) if what == "ffn" else (zero(2 * di, d), None)
    down = one_per_row(L, q8, torch.arange(d, device=DEV) % di, di, dt) if what == "ffn" else zero(d, di)
    ones = torch.ones(d, device=DEV, dtype=dt)
    for kind, w in ((L.W_EMBD, embd), (L.W_ATTN_NORM, ones), (L.W_QKV, qkv), (L.W_O, o), (L.W_FFN_NORM, ones), (L.W_GATE_UP, gu), (L.W_DOWN, down),
                    (L.W_OUT_NORM, ones), (L.W_LM_HEAD, torch.zeros(cfg.vocab, d, device=DEV, dtype=dt))):
        ctx.set_weight(0, kind, w)
    ctx.kv_pool_attach(torch.zeros(128 * ctx.page_bytes // 2, device=DEV, dtype=dt))
    return cfg, ctx, embd, o64 if what == "o" else gu64


def first_tokens(L, ctx, toks):
    """The residual stream after a round of every sequence's first token."""
    out = torch.zeros(len(toks), 2, dtype=torch.int32, device=DEV)
    seqs = [ctx.seq_create() for _ in toks]
    ctx.step([(s, 0, 1) for s in seqs], np.asarray(toks, np.uint32), out)
    x = ctx.hidden(len(toks))
    assert ctx.device_status() == 0
    for s in seqs:
        ctx.seq_free(s)
    return x


def normed(L, x, eps):
    """The library's own norm (the same kernel as in a round), rounded."""
    y = torch.empty_like(x)
    dt = 0 if x.dtype == torch.float16 else 1
    ones = torch.ones(x.shape[1], device=DEV, dtype=x.dtype)
    L.check(L.load_library().lcu_op_rms_norm(y.data_ptr(), x.shape[1], x.data_ptr(), x.shape[1], ones.data_ptr(), dt, eps, x.shape[0], x.shape[1], dt, L.stream_ptr()))
    return y


FORMS = [(0, False), (1, False), (0, True)]  # activations, Q8_0


@pytest.mark.parametrize("act,q8", FORMS)
@pytest.mark.parametrize("n", [3, 9, 16, 17, 33, 48, 64, 100])
@pytest.mark.parametrize("d,nh", [(256, 2), (256, 64), (1280, 10), (4096, 32), (2304, 64)])
@pytest.mark.parametrize("cluster", [0, 2])
def test_output_projection(L, act, q8, n, d, nh, cluster):
    """128 rows and more, 256 to 8192 columns: 1 to 6 pieces of a row block (cluster 0: through scratch; 2: in a cluster wherever there is one)."""
    if q8 and cluster:
        pytest.skip("no cluster form")
    L.set_tuning("tc_cluster", cluster)
    cfg, ctx, embd, w = one_layer(L, act, q8, d, nh, 256, n, "o")
    toks = np.arange(7, 7 + n)
    x = embd[torch.from_numpy(toks).to(DEV)]
    v = normed(L, x, cfg.eps)[:, torch.arange(nh * 128, device=DEV) % d].double()
    want = x.double() + v @ w.T
    got = [first_tokens(L, ctx, toks).double() for _ in range(2)]
    ctx.close()
    # one rounding to the activation dtype, and f32 sums of 2 k + 1 terms in any order
    bound = want.abs() * 2.0 ** (-11 if act == 0 else -8) + (v.abs() @ w.abs().T + x.double().abs()) * (2 * nh * 128 + 1) * 2.0 ** -24
    assert bool(((got[0] - want).abs() <= bound).all())
    assert torch.equal(got[0], got[1])  # tickets were left as they were found


@pytest.mark.parametrize("act,q8", FORMS)
@pytest.mark.parametrize("n", [3, 16, 33, 48, 64])
@pytest.mark.parametrize("d,di", [(512, 256), (4096, 1280), (4096, 6400)])
def test_feed_forward(L, act, q8, n, d, di):
    """SwiGLU of whole and of cut row blocks."""
    L.set_tuning("tc_cluster", 0)
    cfg, ctx, embd, w = one_layer(L, act, q8, d, 2, di, n, "ffn", lambda cfg, g, dt: torch.randn(cfg.vocab, cfg.d, device=DEV, generator=g).mul_(2.0 ** -6).to(dt))
    toks = np.arange(5, 5 + n)
    x = embd[torch.from_numpy(toks).to(DEV)]
    gate, up = (normed(L, x, cfg.eps).double() @ w.T).chunk(2, 1)
    act64 = (torch.nn.functional.silu(gate) * up)[:, torch.arange(d, device=DEV) % di]
    err = first_tokens(L, ctx, toks).double() - x.double() - act64
    ctx.close()
    # gate, up, their product and the sum are rounded: four errors of up to 2^-11 (bf16: 2^-8), a third of which shows in a norm
    assert float(err.norm() / act64.norm()) < 4 / 3 * 2.0 ** (-11 if act == 0 else -8)


@pytest.mark.parametrize("n", [4, 16, 48, 64])
@pytest.mark.parametrize("d,nh", [(256, 64), (4096, 32)])
def test_poisoned_round(L, n, d, nh):
    """Sequences whose embedding holds infinities or a NaN, Q8_0 weights, row blocks cut and whole: they end as with the mma.sync kernel,
    and the others as if the poisoned ones were not there."""
    def embd(cfg, g, dt):
        e = torch.randn(cfg.vocab, cfg.d, device=DEV, generator=g).to(dt)
        e[1], e[2, 7], e[3, ::50] = float("nan"), float("inf"), float("-inf")
        return e
    cfg, ctx, e, w = one_layer(L, 0, True, d, nh, 256, n, "o", embd)
    toks = np.array([1 + i % 3 if i % 4 == 1 else 10 + i for i in range(n)])
    clean = np.where(toks < 4, 9, toks)
    a, b = first_tokens(L, ctx, toks), first_tokens(L, ctx, clean)
    good = torch.from_numpy(toks >= 4).to(DEV)
    assert torch.equal(a[good], b[good]) and bool(b.isfinite().all())
    L.set_tuning("tc", 0, ctx)
    c = first_tokens(L, ctx, toks)
    assert torch.equal(a.isnan(), c.isnan()) and torch.equal(a.isinf(), c.isinf())
    assert bool(a[~good].isnan().any())
    ctx.close()


@pytest.mark.parametrize("family", ["zefedra", "galarax", "mupuvik", "gunulorn"])
def test_layered_prompt(L, family):
    """A prompt of more than 128 tokens: f32 rows, xIELU, squared ReLU, gated units and capped logits with and without the 256-row tiles."""
    M = importlib.import_module(family + "_models")
    raw = M.MIXED
    w = M.weights(raw, 3)
    toks = M.random_tokens(raw, 200, 4)
    got = []
    for v in (0, 1):
        L.set_tuning("tc_pair_min", v)
        cfg, ctx = M.load(L, raw, w, 1)
        out = torch.zeros(1, 2, dtype=torch.int32, device=DEV)
        rows = ctx.step_logits([(ctx.seq_create(), 0, 200)], np.asarray(toks, np.uint32), list(range(0, 200, 3)))
        got.append(rows.double().cpu())
        assert ctx.device_status() == 0
        ctx.close()
    # sums in another order: roundings of the activations that end up on the other side
    assert float((got[0] - got[1]).norm() / got[0].norm()) <= 2.5e-2
    assert got[1].isfinite().all()
