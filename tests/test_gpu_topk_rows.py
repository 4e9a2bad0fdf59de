"""Per-contig selection: rows around the 32, 256 and 512 entries of its register
forms, limits around the sizes of its sorts, equal scores inside the kept set
and at its border, scores over a wide range.  Expected: the same edges taken by
numpy from the list that a limit above every row length gives (another kernel)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))

pytestmark = pytest.mark.gpu


def _rows(n, kind, seed):
    rng = np.random.default_rng(seed)
    c = np.repeat(rng.dirichlet(np.full(136, 8.0))[None] * 4000.0, n, 0)
    c = c + rng.uniform(0, 40 if kind == "wide" else 6, (n, 136))
    ln = rng.uniform(20000, 500000, n)
    if kind == "ties":  # groups of five equal contigs
        c, ln = c[np.arange(n) // 5 * 5 % n], ln[np.arange(n) // 5 * 5 % n]
        at = rng.permutation(n)
        c, ln = c[at], ln[at]
    tnf = (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32)
    return tnf, np.log10(ln)


def _run(torch, ctx, d_tnf, d_ls, n, cutoff, k, cap):
    fr, to = (torch.zeros(cap, dtype=torch.int64, device="cuda") for _ in range(2))
    st = torch.zeros(cap, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    m, _ = ctx.tnf_graph_dev(d_tnf.data_ptr(), d_ls.data_ptr(), n, cutoff, k, "plain", fr.data_ptr(), to.data_ptr(),
                             st.data_ptr(), cap)
    return fr[:m].cpu().numpy(), to[:m].cpu().numpy(), st[:m].cpu().numpy()


@pytest.mark.parametrize("n", [2, 32, 33, 34, 257, 258, 513, 514, 700])
@pytest.mark.parametrize("kind", ["plain", "ties", "wide"])
def test_selection_equals_sorted_rows(gpu_ctx, n, kind):
    torch = pytest.importorskip("torch")

    tnf, ls = _rows(n, kind, n)
    d_tnf, d_ls = torch.from_numpy(tnf).cuda(), torch.from_numpy(ls).cuda()
    cutoff = 0.05 if kind == "wide" else 0.5
    f, t, s = _run(torch, gpu_ctx, d_tnf, d_ls, n, cutoff, 4096, n * n)
    if kind != "wide":
        assert len(f) == n * (n - 1) // 2
    sim = np.full((n, n), -1.0)
    sim[f, t] = s
    sim[t, f] = s
    for k in (1, 2, 31, 32, 33, 64, 65, 128, 129, 200, 256, 257, 512):
        want = []
        for i in range(n):
            order = np.lexsort((np.arange(n), -sim[i]))[:k]
            want += [(i, int(j), float(sim[i, j])) for j in order if j > i and sim[i, j] >= 0]
        got = _run(torch, gpu_ctx, d_tnf, d_ls, n, cutoff, k, n * min(n, k))
        assert list(zip(*(a.tolist() for a in got))) == want
