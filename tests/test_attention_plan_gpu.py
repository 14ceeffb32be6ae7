"""The split of attention in decode rounds follows the longest context: rounds that cross its steps, captured and eager, against the
same tokens as one prompt."""
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n_seq", [1, 2, 5, 40])
@pytest.mark.parametrize("dh,nkvh", [(64, 2), (128, 1)])
@pytest.mark.parametrize("start", [1, 126, 510])
def test_growing_contexts(L, n_seq, dh, nkvh, start):
    cfg = replace(L.CONFIGS["tiny"], d=256, nh=4, nkvh=nkvh, dh=dh, di=512, nctx=1024)
    w = L.synth_weights_numpy(cfg, 3)
    rng = np.random.default_rng(start + n_seq)
    lens = [start if i == 0 else 1 + (start * (i % 7)) // 8 for i in range(n_seq)]
    toks = [rng.integers(3, cfg.vocab, n + 5).astype(np.uint32) for n in lens]
    stream = torch.cuda.Stream(device=DEV)
    got = []
    for graph in (1, 0):
        ctx = L.load_model(cfg, w, kv_bytes=256 << 20)
        ctx.set_cuda_graph(graph)
        out = torch.zeros(n_seq, 2, dtype=torch.int32, device=DEV)
        seqs = [ctx.seq_create() for _ in toks]
        for s, t, n in zip(seqs, toks, lens):
            ctx.step([(s, 0, n)], t[:n], out, stream=stream)
        rows = []
        for k in range(5):
            ctx.step([(s, n + k, 1) for s, n in zip(seqs, lens)], np.array([t[n + k] for t, n in zip(toks, lens)], np.uint32), out, stream=stream)
            rows.append(ctx.logits(n_seq))
        got.append(torch.stack(rows))
        if not graph:
            whole = []
            for t in toks:
                s = ctx.seq_create()
                ctx.step([(s, 0, len(t))], t, out, stream=stream)
                whole.append(ctx.logits(1)[0])
                ctx.seq_free(s)
        assert ctx.device_status() == 0
        ctx.close()
    assert torch.equal(got[0], got[1])
    a, b = got[0][-1].double(), torch.stack(whole).double()
    assert float((a - b).norm() / b.norm()) < 3e-3  # sums in another order: a few roundings end up on the other side
