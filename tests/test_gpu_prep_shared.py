"""Scoring given pairs between two graphs of one assembly leaves the graph's
preparation in place, whatever its order, and scores as it does by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 9000])  # ordered by size; in bands
def test_pair_scores_between_graphs(n):
    torch = pytest.importorskip("torch")
    import mdet_gb300 as m

    rng = np.random.default_rng(n)
    g = rng.integers(0, 20, n)
    c = rng.dirichlet(np.full(136, 2.0), 20)[g] * 4000.0 + rng.uniform(0, 20, (n, 136))
    tnf = torch.from_numpy((c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32)).cuda()
    ls = torch.from_numpy(np.log10(rng.uniform(2500, 500000, n))).cuda()
    pairs = torch.from_numpy(rng.integers(0, n, (5000, 2))).cuda()
    out = [torch.zeros(n * 50, dtype=t, device="cuda") for t in (torch.int64, torch.int64, torch.float64)]
    torch.cuda.synchronize()

    def graph(ctx):
        k, st = ctx.tnf_graph_dev(tnf.data_ptr(), ls.data_ptr(), n, 0.9, 50, "bf16", *(x.data_ptr() for x in out), n * 50)
        return st["gpu_launches"], [x[:k].clone() for x in out]

    def scores(ctx):
        d, p = (torch.zeros(5000, dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        ctx.pair_scores_dev(tnf.data_ptr(), ls.data_ptr(), n, pairs.data_ptr(), 5000, d.data_ptr(), p.data_ptr())
        return d, p

    with m.Context(0) as alone, m.Context(0) as both:
        want = scores(alone)
        graph(both)
        scores(both)
        graph(both)  # buffers in place: from here on a preparation that is kept is used
        launches, edges = graph(both)
        got = scores(both)
        again, same = graph(both)
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    assert again == launches and all(torch.equal(a, b) for a, b in zip(edges, same))
