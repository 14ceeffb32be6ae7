"""Q8_0 linear layers on tcgen05: weights as pairs of f16, up to 64 tokens a pass and in 256-row tiles on pairs of SMs, against f64."""
import ctypes as C
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def product(L, n, out, k, scales, seed, x_scale=1.0, res=True):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    x = (torch.randn(n, k, device=DEV, generator=g) * x_scale).half()
    q = torch.randint(-128, 128, (out, k), dtype=torch.int8, device=DEV, generator=g)
    lo, hi = scales
    s = torch.exp(torch.empty(out, k // 32, device=DEV).uniform_(np.log(lo), np.log(hi), generator=g)).half()
    r = torch.randn(n, out, device=DEV, generator=g).half() if res else None
    w = torch.cat([q.view(torch.uint8).reshape(-1), s.view(torch.uint8).reshape(-1)])
    y = torch.full((n + 1, out), 7.0, device=DEV, dtype=torch.float16)
    L.check(L.load_library().lcu_op_linear(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), L.Q8_0, r.data_ptr() if res else None, out, n, k, out, 0,
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    wd = (q.double().view(out, -1, 32) * s.double()[..., None]).view(out, k)
    want = x.double() @ wd.T + (r.double() if res else 0)
    # one rounding to f16 (subnormal results: half of 2^-24), and f32 sums of 2 k + 1 terms in any order
    bound = want.abs() * 2.0 ** -11 + 2.0 ** -25 + (x.double().abs() @ wd.abs().T + (r.double().abs() if res else 0)) * (2 * k + 1) * 2.0 ** -24
    ok = (y[:n].double() - want).abs() <= bound
    return bool((ok | (want.abs() > 65000)).all()) and bool((y[n:] == 7.0).all())


@pytest.mark.parametrize("n", [5, 16, 17, 33, 48, 49, 64, 65, 100, 129, 256, 300, 520])
@pytest.mark.parametrize("out,k", [(2, 256), (130, 512), (136, 2816), (1000, 768), (4096, 1280), (9480, 256), (19200, 512)])
def test_product(L, n, out, k):
    assert product(L, n, out, k, (1e-4, 4e-4), n * out + k)


@pytest.mark.parametrize("n", [7, 40, 300])
@pytest.mark.parametrize("scales,x_scale", [((6e-8, 1e-6), 1.0), ((1e-6, 1e-2), 1.0), ((100.0, 60000.0), 1e-5)])
def test_scales(L, n, scales, x_scale):
    """Subnormal scales (the low halves are subnormal f16 numbers), scales far apart, and products beyond the range of f16."""
    assert product(L, n, 264, 512, scales, n, x_scale, res=False)


def linear(L, x, w, y, r=None):
    n, k = x.shape
    out = y.shape[1]
    L.check(L.load_library().lcu_op_linear(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), L.Q8_0, r.data_ptr() if r is not None else None, out, n, k, out, 0,
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))


def planes(q, s):
    return torch.cat([q.view(torch.uint8).reshape(-1), s.view(torch.uint8).reshape(-1)])


def poison(x, kind):
    """Activations that are not finite, as an overflow in an earlier layer leaves them."""
    k, inf = x.shape[-1], float("inf")
    if kind == "nan":
        x[:] = float("nan")
    elif kind == "zeros and a late nan":  # a norm of a row that holds an infinity
        x[:] = 0
        x[..., k - 7] = float("nan")
    elif kind == "an infinity":
        x[..., 37] = inf
    elif kind == "infinities of both signs":
        x[..., k - 3], x[..., k - 40] = inf, -inf
    elif kind == "infinities of one sign":
        x[..., 5::97] = -inf
    elif kind == "infinite":
        x[:] = inf
    return x


KINDS = ["finite", "nan", "zeros and a late nan", "an infinity", "infinities of both signs", "infinities of one sign", "infinite"]


@pytest.mark.parametrize("n", [7, 16, 40, 64, 100, 300])
@pytest.mark.parametrize("out,k", [(2, 256), (130, 512), (136, 2816), (1000, 768)])
@pytest.mark.parametrize("res", [False, True])
def test_not_finite(L, n, out, k, res):
    """Infinities and NaN among the activations and the scales, and scales whose products leave the range of f16, mixed with finite rows:
    the same values as the mma.sync kernel's."""
    g = torch.Generator(device=DEV)
    g.manual_seed(n * out + k)
    x = torch.randn(n, k, device=DEV, generator=g).mul_(0.1).half()
    for i in range(n):
        poison(x[i], KINDS[i % 8 % 7] if i % 3 or i < 7 else "finite")
    q = torch.randint(-128, 128, (out, k), dtype=torch.int8, device=DEV, generator=g)
    q[:, 37] *= torch.arange(out, device=DEV) % 5 != 0  # zero times infinity
    s = torch.empty(out, k // 32, device=DEV).uniform_(1e-4, 4e-4, generator=g).half()
    for row, v in ((0, 30000.0), (1, 0.0), (5, float("inf")), (6, float("nan")), (77, 600.0)):
        if row < out:
            s[row, (k // 32 - 1) // 2] = v
    r = torch.randn(n, out, device=DEV, generator=g).half() if res else None
    got = []
    try:
        for tc in (0, 1):
            L.set_tuning("tc", tc)
            y = torch.full((n + 1, out), 7.0, device=DEV, dtype=torch.float16)
            linear(L, x, planes(q, s), y, r)
            assert bool((y[n:] == 7.0).all())
            got.append(y[:n].double())
    finally:
        L.set_tuning("tc", 1)
    a, b = got
    assert torch.equal(a.isnan(), b.isnan())
    assert torch.equal(a.isinf() * a.sign().nan_to_num(), b.isinf() * b.sign().nan_to_num())
    fin = a.isfinite()
    wd = (q.double().view(out, -1, 32) * s.double()[..., None]).view(out, k)
    # two roundings to f16 and two f32 sums of 2 k + 1 terms in any order
    bound = a.abs() * 2.0 ** -10 + 2.0 ** -24 + (x.double().abs() @ wd.abs().T + (r.double().abs() if res else 0)) * (2 * k + 1) * 2.0 ** -23
    assert bool(((a - b).abs() <= bound)[fin].all())


@pytest.mark.parametrize("n", [16, 64, 500])
@pytest.mark.parametrize("kind", KINDS[1:])
def test_not_finite_in_time(L, n, kind):
    """A token that is not finite does not hold up the others of its round (one thread per product took 30 to 1000 times as long)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(n)
    out, k = 8192, 4096
    q = torch.randint(-128, 128, (out, k), dtype=torch.int8, device=DEV, generator=g)
    w = planes(q, torch.empty(out, k // 32, device=DEV).uniform_(1e-4, 4e-4, generator=g).half())
    y = torch.empty(n, out, device=DEV, dtype=torch.float16)

    def best(x):
        times = []
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            linear(L, x, w, y)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        return min(times)
    x = torch.randn(n, k, device=DEV, generator=g).half()
    base = best(x)
    one, every = x.clone(), x.clone()
    poison(one[n // 2], kind)
    poison(every, kind)
    assert best(one) < 3 * base
    assert best(every) < (4 if "nan" in kind else 25) * base


@pytest.mark.parametrize("n", [3, 40, 64, 130, 300])
def test_round(L, n):
    """RoPE with cache append, residual and SwiGLU of a round: the same prompt with the mma.sync kernel."""
    cfg = replace(L.CONFIGS["tiny"], d=512, nh=8, nkvh=2, dh=64, di=1280, weight_dtype=L.Q8_0, nctx=1024)
    w = L.synth_weights_numpy(cfg, 3)
    prompt = np.random.default_rng(n).integers(3, cfg.vocab, n).astype(np.uint32)
    got = []
    try:
        for v in (0, 1):
            L.set_tuning("tc", v)
            ctx = L.load_model(cfg, w)
            out = torch.zeros(1, 2, dtype=torch.int32, device=DEV)
            s = ctx.seq_create()
            ctx.step([(s, 0, n)], prompt, out)
            ctx.step([(s, n, 1)], prompt[:1], out)  # reads the cache that the prompt left
            got.append((ctx.hidden(1).double(), ctx.logits(1).double()))
            assert ctx.device_status() == 0
            ctx.close()
    finally:
        L.set_tuning("tc", 1)
    for a, b in zip(*got):  # sums in another order: a few roundings of the activations end up on the other side
        assert float((a - b).norm() / b.norm()) < 3e-3
