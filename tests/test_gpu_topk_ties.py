"""Per-contig selection with equal scores -- pairs, groups around the 32 that a lane
each holds, whole rows -- at the border of the kept set and inside it, and rows around
the 512, 880 and 1,024 entries that are staged.  Expected: the same edges taken by
numpy from the list that a limit above every row length gives (another kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, group, seed):
    rng = np.random.default_rng(seed)
    c = np.repeat(rng.dirichlet(np.full(136, 8.0))[None] * 4000.0, n, 0) + rng.uniform(0, 6, (n, 136))
    ln = rng.uniform(20000, 500000, n)
    at = rng.permutation(n) // group * group  # equal contigs lie apart
    c, ln = c[at], ln[at]
    return (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32), np.log10(ln)


def _run(torch, ctx, d_tnf, d_ls, n, k):
    cap = n * min(n, k)
    fr, to = (torch.zeros(cap, dtype=torch.int64, device="cuda") for _ in range(2))
    st = torch.zeros(cap, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    m, _ = ctx.tnf_graph_dev(d_tnf.data_ptr(), d_ls.data_ptr(), n, 0.5, k, "plain", fr.data_ptr(), to.data_ptr(),
                             st.data_ptr(), cap)
    return fr[:m].cpu().numpy(), to[:m].cpu().numpy(), st[:m].cpu().numpy()


@pytest.mark.parametrize("n,group", [(300, 2), (300, 20), (300, 31), (300, 33), (300, 64), (300, 300), (513, 2),
                                     (514, 40), (600, 600), (870, 5), (880, 20), (881, 3), (881, 881), (882, 17),
                                     (1024, 6), (1025, 33), (1026, 2)])
def test_equal_scores(gpu_ctx, n, group):
    torch = pytest.importorskip("torch")
    tnf, ls = _rows(n, group, n + group)
    d_tnf, d_ls = torch.from_numpy(tnf).cuda(), torch.from_numpy(ls).cuda()
    f, t, s = _run(torch, gpu_ctx, d_tnf, d_ls, n, 4096)
    assert len(f) == n * (n - 1) // 2
    sim = np.full((n, n), -1.0)
    sim[f, t] = s
    sim[t, f] = s
    order = np.argsort(-sim, axis=1, kind="stable")  # equal scores by column; the diagonal last
    for k in (1, 31, 33, 64, 127, 200, 256, 257, 400, 512):
        i = np.repeat(np.arange(n), min(k, n - 1))
        j = order[:, :min(k, n - 1)].ravel()
        keep = j > i
        i, j = i[keep], j[keep]
        got = _run(torch, gpu_ctx, d_tnf, d_ls, n, k)
        assert np.array_equal(got[0], i) and np.array_equal(got[1], j) and np.array_equal(got[2], sim[i, j])
