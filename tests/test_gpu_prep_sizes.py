"""Preparation at its edges: contig counts around the 64- and 256-row blocks, TNF
rows on a 4-byte boundary (scalar loads) as on a 16-byte one, log sizes out of
order and tied, and several sets prepared together."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    centre = rng.dirichlet(np.full(136, 8.0), 3)
    c = rng.poisson(centre[rng.integers(0, 3, n)] * 4000.0).astype(np.float64)
    tnf = (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32)
    ls = np.log10(rng.choice([2500.0, 4000.0, 9000.0, 61234.0, 500000.0], n))
    return tnf, ls


def _dev(torch, tnf, ls, shift):
    n = tnf.shape[0]
    buf = torch.zeros(n * 136 + 8, dtype=torch.float32, device="cuda")
    view = buf[shift:shift + n * 136]
    view.copy_(torch.from_numpy(tnf.ravel()))
    return buf, view, torch.from_numpy(ls).cuda()


@pytest.mark.parametrize("n", [2, 63, 64, 65, 255, 256, 257, 1100])
@pytest.mark.parametrize("mode", ["bf16", "tf32", "plain"])
def test_graph_sizes_and_alignment(gpu_ctx, n, mode):
    torch = pytest.importorskip("torch")
    from oracle import oracle

    tnf, ls = _rows(n, n)
    of, ot, os_ = oracle.graph(tnf, ls, 0.9, 50)
    for shift in (0, 1, 3):
        buf, view, d_ls = _dev(torch, tnf, ls, shift)
        cap = n * 50
        fr, to = (torch.zeros(cap, dtype=torch.int64, device="cuda") for _ in range(2))
        st = torch.zeros(cap, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        k, _ = gpu_ctx.tnf_graph_dev(view.data_ptr(), d_ls.data_ptr(), n, 0.9, 50, mode, fr.data_ptr(),
                                     to.data_ptr(), st.data_ptr(), cap)
        got = dict(zip(zip(fr[:k].tolist(), to[:k].tolist()), st[:k].tolist()))
        ref = dict(zip(zip(of.tolist(), ot.tolist()), os_.tolist()))
        # the exact stage's probability is within 1e-9 of FP64; no pair here lies that near a decision
        assert got.keys() == ref.keys()
        assert all(abs(got[e] - ref[e]) < 1e-9 for e in ref)


def test_batch_of_edge_sizes(gpu_ctx):
    torch = pytest.importorskip("torch")

    sizes = [2, 257, 1, 256, 70, 0, 513]
    items, keep = [], []
    for i, n in enumerate(sizes):
        tnf, ls = _rows(max(n, 1), 40 + i)
        buf, view, d_ls = _dev(torch, tnf, ls, i % 2)
        out = [torch.zeros(max(1, n * 50), dtype=t, device="cuda")
               for t in (torch.int64, torch.int64, torch.float64)]
        keep.append((buf, d_ls, out, view))
        items.append(dict(d_tnf=view.data_ptr(), d_ls=d_ls.data_ptr(), n=n, cutoff=0.9 if i % 3 else 0.95,
                          max_edges=50, d_from=out[0].data_ptr(), d_to=out[1].data_ptr(),
                          d_stnf=out[2].data_ptr(), capacity=out[0].numel()))
    torch.cuda.synchronize()
    res, _ = gpu_ctx.tnf_graph_batched(items, "bf16")
    for n, it, (buf, d_ls, out, view), (status, k) in zip(sizes, items, keep, res):
        assert status == 0
        if n < 2:
            assert k == 0
            continue
        one = [torch.zeros_like(o) for o in out]
        torch.cuda.synchronize()
        k1, _ = gpu_ctx.tnf_graph_dev(it["d_tnf"], it["d_ls"], n, it["cutoff"], 50, "bf16", one[0].data_ptr(),
                                      one[1].data_ptr(), one[2].data_ptr(), one[0].numel())
        assert k1 == k
        for a, b in zip(out, one):
            assert torch.equal(a[:k], b[:k])
