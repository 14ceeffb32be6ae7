"""Attention of prompts on tcgen05: tiles of rows and positions, page sizes and groups of heads, against the mma.sync kernel and f64."""
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def form(L):
    yield lambda v: L.set_tuning("attn_tc", v)
    L.set_tuning("attn_tc", 1)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("nh,nkvh,dh,page", [(4, 4, 64, 8), (4, 2, 128, 16), (8, 2, 64, 64), (8, 1, 128, 128), (4, 1, 64, 32)])
@pytest.mark.parametrize("past,n", [(0, 2), (0, 33), (0, 128), (1, 129), (127, 64), (5, 300), (250, 257), (0, 640)])
def test_round(L, form, act, nh, nkvh, dh, page, past, n):
    """A prompt of which `past` tokens are cached, beside two running sequences; the pages hold NaN where nothing was written."""
    cfg = replace(L.CONFIGS["tiny"], d=256, nh=nh, nkvh=nkvh, dh=dh, di=512, act_dtype=act, nctx=1024)
    w = L.synth_weights_numpy(cfg, 3)
    rng = np.random.default_rng(n + past)
    toks = rng.integers(3, cfg.vocab, past + n + 200).astype(np.uint32)
    got = []
    for v in (0, 2):
        form(v)
        ctx = L.Context(cfg.desc(page), 0)
        keep = []
        for (layer, kind), t in w.items():
            t = torch.from_numpy(t.view(np.int16)).to(DEV)
            keep.append(t)
            ctx.set_weight(max(layer, 0), kind, t)
        pool = torch.full((((past + n) // page + 200 // page + 6) * ctx.page_bytes // 2,), float("nan"), device=DEV, dtype=L.torch_dtype(act))
        ctx.kv_pool_attach(pool)
        out = torch.zeros(3, 2, dtype=torch.int32, device=DEV)
        a, b, p = ctx.seq_create(), ctx.seq_create(), ctx.seq_create()
        ctx.step([(a, 0, 1)], toks[:1], out)
        ctx.step([(b, 0, 150)], toks[:150], out)
        if past:
            ctx.step([(p, 0, past)], toks[:past], out)
        ctx.step([(a, 1, 1), (p, past, n), (b, 150, 1)], np.concatenate([toks[1:2], toks[past:past + n], toks[150:151]]), out)
        got.append((ctx.hidden(n + 2).double(), ctx.logits(3).double()))
        assert ctx.device_status() == 0
        ctx.close()
    for x, y in zip(*got):  # sums in another order: a few roundings of the activations end up on the other side
        assert float((x - y).norm() / y.norm()) < (2e-3 if act == 0 else 1.5e-2)


@pytest.mark.parametrize("dh,nh", [(64, 4), (128, 8)])
def test_against_f64(L, form, dh, nh):
    """One layer whose output projection is the identity: the attention of every token of a prompt, against f64."""
    n, d = 517, nh * dh
    cfg = replace(L.CONFIGS["tiny"], n_layers=1, d=d, nh=nh, nkvh=nh // 4, dh=dh, di=64, nctx=1024)
    w = L.synth_weights_numpy(cfg, 5)
    w[(0, L.W_O)] = np.eye(d, dtype=np.float16).view(w[(0, L.W_O)].dtype)
    w[(0, L.W_DOWN)] = np.zeros_like(w[(0, L.W_DOWN)])
    w[(0, L.W_QKV)] = (w[(0, L.W_QKV)].view(np.float16) * np.float16(3)).view(w[(0, L.W_QKV)].dtype)
    toks = np.random.default_rng(1).integers(3, cfg.vocab, n).astype(np.uint32)

    def f64(kind):
        return torch.from_numpy(w[(0, kind) if (0, kind) in w else (-1, kind)].view(np.float16).astype(np.float64)).to(DEV)
    x = f64(L.W_EMBD)[torch.from_numpy(toks.astype(np.int64)).to(DEV)]
    h = x / torch.sqrt((x * x).mean(-1, keepdim=True) + cfg.eps) * f64(L.W_ATTN_NORM)
    q, k, v = (h @ f64(L.W_QKV).T).split([d, d // 4, d // 4], 1)
    ang = torch.arange(n, device=DEV).double()[:, None] * cfg.theta ** (-torch.arange(0, dh, 2, device=DEV).double() / dh)

    def rot(t):
        a, b = t.view(n, -1, dh)[..., 0::2], t.view(n, -1, dh)[..., 1::2]
        c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    q, k, v = rot(q), rot(k).repeat_interleave(4, 1), v.view(n, -1, dh).repeat_interleave(4, 1)
    s = torch.einsum("ihd,jhd->hij", q, k) * dh ** -0.5
    s = s.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=DEV).tril(), float("-inf"))
    want = x + torch.einsum("hij,jhd->ihd", torch.softmax(s, -1), v).reshape(n, d)
    err = []
    for on in (0, 2):
        form(on)
        ctx = L.load_model(cfg, w)
        out = torch.zeros(1, 2, dtype=torch.int32, device=DEV)
        ctx.step([(ctx.seq_create(), 0, n)], toks, out)
        err.append(float((ctx.hidden(n).double() - want).norm() / want.norm()))
        ctx.close()
    assert err[1] < 2e-3 and err[1] <= 1.05 * err[0] + 1e-6, err
