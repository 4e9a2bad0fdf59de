"""The exact stage's edge queues: sets in which every pair is an edge (each warp's
queue fills at 32 a round) or none is, at pair counts around a warp's 32, a
block's 256 and a queue's 96, and pairs whose rows differ in the last columns
only."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))

pytestmark = pytest.mark.gpu


def _rows(n, spread, seed):
    rng = np.random.default_rng(seed)
    c = rng.dirichlet(np.full(136, 8.0)) * 4000.0
    c = np.repeat(c[None], n, 0)
    if spread == "none":
        c = rng.dirichlet(np.full(136, 0.3), n) * 4000.0
    elif spread == "tail":
        c[:, 128:] += rng.uniform(0, 30, (n, 8))
    else:
        c += rng.uniform(0, 4, (n, 136))
    tnf = (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32)
    return tnf, np.log10(rng.uniform(20000, 500000, n))


@pytest.mark.parametrize("n", [2, 8, 9, 14, 23, 24, 100, 300])
@pytest.mark.parametrize("spread", ["all", "tail", "none"])
def test_every_or_no_pair(gpu_ctx, n, spread):
    torch = pytest.importorskip("torch")
    from oracle import oracle

    tnf, ls = _rows(n, spread, n)
    of, ot, os_ = oracle.graph(tnf, ls, 0.9, 500)
    ref = dict(zip(zip(of.tolist(), ot.tolist()), os_.tolist()))
    assert spread == "tail" or len(ref) == (0 if spread == "none" else n * (n - 1) // 2)
    d_tnf, d_ls = torch.from_numpy(tnf).cuda(), torch.from_numpy(ls).cuda()
    for mode in ("bf16", "tf32", "plain"):
        cap = n * 500
        fr, to = (torch.zeros(cap, dtype=torch.int64, device="cuda") for _ in range(2))
        st = torch.zeros(cap, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        k, _ = gpu_ctx.tnf_graph_dev(d_tnf.data_ptr(), d_ls.data_ptr(), n, 0.9, 500, mode, fr.data_ptr(),
                                     to.data_ptr(), st.data_ptr(), cap)
        got = dict(zip(zip(fr[:k].tolist(), to[:k].tolist()), st[:k].tolist()))
        assert got.keys() == ref.keys()
        assert all(abs(got[e] - ref[e]) < 1e-9 for e in ref)
