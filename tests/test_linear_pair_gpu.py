"""The 256-row tiles on pairs of SMs: edges of tiles and remainders against f64 products, and every epilogue of a round against the
kernels of smaller rounds."""
import ctypes as C
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def pair(L):
    """Sets the fewest tokens that take the tiles (0: none does)."""
    yield lambda v: L.set_tuning("tc_pair_min", v)
    L.set_tuning("tc_pair_min", 129)


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("n", [9, 127, 129, 256, 257, 520])
@pytest.mark.parametrize("out,k", [(8, 64), (136, 512), (1000, 192), (4096, 448), (9480, 960)])
@pytest.mark.parametrize("res", [False, True])
def test_product(L, pair, dt, n, out, k, res):
    pair(1)
    tdt = L.torch_dtype(dt)
    g = torch.Generator(device=DEV)
    g.manual_seed(n * out + k)
    x = torch.randn(n, k, device=DEV, generator=g).to(tdt)
    w = torch.randn(out, k, device=DEV, generator=g).to(tdt)
    r = torch.randn(n, out, device=DEV, generator=g).to(tdt) if res else None
    y = torch.full((n + 1, out), 7.0, device=DEV, dtype=tdt)
    L.check(L.load_library().lcu_op_linear(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), dt, r.data_ptr() if res else None, out, n, k, out, dt,
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want = x.double() @ w.double().T + (r.double() if res else 0)
    # one rounding to the activation dtype, and f32 sums of k + 1 terms in any order
    bound = want.abs() * 2.0 ** (-11 if dt == 0 else -8) + (x.double().abs() @ w.double().abs().T + 1) * (k + 1) * 2.0 ** -24
    assert bool(((y[:n].double() - want).abs() <= bound).all())
    assert bool((y[n:] == 7.0).all())


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("n,out,k", [(200, 6144, 4096), (300, 4096, 4096), (300, 4096, 14336), (1000, 2048, 8192), (520, 1024, 1088)])
def test_sums(L, pair, dt, n, out, k):
    """The tensor pipe cuts a sum off where it would have to round it: an error that grows with the products of one accumulator.  Sums
    are cut into as many pieces as CTAs would fill the GPU with.  Seen by way of a residual that takes the rounded product away again."""
    pair(1)
    tdt = L.torch_dtype(dt)
    g = torch.Generator(device=DEV)
    g.manual_seed(k)
    x = torch.randn(n, k, device=DEV, generator=g).to(tdt)
    w = torch.randn(out, k, device=DEV, generator=g).mul_(0.02).to(tdt)
    want = x.double() @ w.double().T
    r = (-want).to(tdt)
    y = torch.empty(n, out, device=DEV, dtype=tdt)
    L.check(L.load_library().lcu_op_linear(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), dt, r.data_ptr(), out, n, k, out, dt,
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    err = y.double() - (want + r.double())
    pieces = min(8, max(1, torch.cuda.get_device_properties(0).multi_processor_count // -(-out // 128)))
    if k // 64 < 32:
        pieces = 1
    while pieces > 1 and k // 64 // pieces < 4:
        pieces -= 1
    steps = -(-k // 64 // pieces) * 4
    # a step of 16 products cuts half a unit of 24 bits on average, of a sum that grows like a root: a third of one of the result; with 30 %
    # to spare.  And y's own rounding, of a difference of 2^-12 (bf16: 2^-9)
    assert float(err.norm() / want.norm()) < 1.3 * steps * 2.0 ** -24 / 3 + (2.0 ** -24 if dt == 0 else 2.0 ** -18)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("n", [130, 300, 513])
def test_round(L, pair, act, n):
    """RoPE with cache append, residual and SwiGLU: the same prompt with and without the tiles."""
    cfg = replace(L.CONFIGS["tiny"], d=512, nh=8, nkvh=2, dh=64, di=1088, act_dtype=act, nctx=1024)
    w = L.synth_weights_numpy(cfg, 3)
    prompt = np.random.default_rng(n).integers(3, cfg.vocab, n).astype(np.uint32)
    got = []
    for v in (0, 1):
        pair(v)
        ctx = L.load_model(cfg, w)
        out = torch.zeros(1, 2, dtype=torch.int32, device=DEV)
        s = ctx.seq_create()
        ctx.step([(s, 0, n)], prompt, out)
        ctx.step([(s, n, 1)], prompt[:1], out)  # reads the cache that the prompt left
        got.append((ctx.hidden(1).double(), ctx.logits(1).double()))
        assert ctx.device_status() == 0
        ctx.close()
    for a, b in zip(*got):  # sums in another order: a few roundings of the activations end up on the other side
        assert float((a - b).norm() / b.norm()) < (3e-3 if act == 0 else 2e-2)
