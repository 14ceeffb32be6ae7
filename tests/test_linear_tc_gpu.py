"""Linear layers of 9 to 128 tokens on tcgen05 as the stand-alone operator runs them, against f64 products: 1 to 300 row blocks, which the
cost rule gives to clusters of 1 to 8 CTAs or to whole row blocks.  The operator has no scratch, so row blocks are never cut here:
those are in test_linear_round_gpu.py."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("n", [9, 16, 33, 64, 65, 128])
@pytest.mark.parametrize("blocks,k", [(1, 64), (3, 2048), (15, 2048), (16, 4096), (20, 2048), (22, 1536), (26, 1280), (33, 1024), (45, 832), (48, 2112),
                                      (75, 1024), (130, 512), (150, 320), (300, 256)])
def test_product(L, dt, n, blocks, k):
    out = blocks * 128 - (56 if blocks % 2 else 0)
    tdt = L.torch_dtype(dt)
    g = torch.Generator(device=DEV)
    g.manual_seed(n * out + k)
    x = torch.randn(n, k, device=DEV, generator=g).to(tdt)
    w = torch.randn(out, k, device=DEV, generator=g).to(tdt)
    r = torch.randn(n, out, device=DEV, generator=g).to(tdt)
    y = torch.full((n + 1, out), 7.0, device=DEV, dtype=tdt)
    L.check(L.load_library().lcu_op_linear(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), dt, r.data_ptr(), out, n, k, out, dt,
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want = x.double() @ w.double().T + r.double()
    # one rounding to the activation dtype, and f32 sums of k + 1 terms in any order
    bound = want.abs() * 2.0 ** (-11 if dt == 0 else -8) + (x.double().abs() @ w.double().abs().T + 1) * (k + 1) * 2.0 ** -24
    assert bool(((y[:n].double() - want).abs() <= bound).all())
    assert bool((y[n:] == 7.0).all())
