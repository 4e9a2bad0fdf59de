"""The tile-shape tuner keeps a batch's lists and the kept tiles of one large graph
apart: after a batch of as many rows, the first graph of a context still times its
own shapes, and the other way round; edges as in a context that ran nothing else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ME = 50


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    g = rng.integers(0, max(3, n // 450), n)
    c = rng.dirichlet(np.full(136, 2.0), g.max() + 1)[g] * 4000.0 + rng.uniform(0, 20, (n, 136))
    return (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32), np.log10(rng.uniform(2500, 500000, n))


class _Calls:
    def __init__(self, torch, sets):
        self.torch = torch
        self.sets = [(torch.from_numpy(t).cuda(), torch.from_numpy(l).cuda(), l.size) for t, l in sets]

    def out(self, n):
        z = self.torch.zeros
        return [z(n * ME, dtype=t, device="cuda") for t in (self.torch.int64, self.torch.int64, self.torch.float64)]

    def graph(self, ctx):
        t, l, n = self.sets[0]
        o = self.out(n)
        self.torch.cuda.synchronize()
        k, st = ctx.tnf_graph_dev(t.data_ptr(), l.data_ptr(), n, 0.9, ME, "bf16", *(x.data_ptr() for x in o), n * ME)
        return st["gpu_launches"], [x[:k].clone() for x in o]

    def batch(self, ctx):
        outs = [self.out(n) for _, _, n in self.sets[1:]]
        self.torch.cuda.synchronize()
        res, st = ctx.tnf_graph_batched(
            [dict(d_tnf=t.data_ptr(), d_ls=l.data_ptr(), n=n, cutoff=0.9, max_edges=ME, d_from=o[0].data_ptr(),
                  d_to=o[1].data_ptr(), d_stnf=o[2].data_ptr(), capacity=n * ME)
             for (t, l, n), o in zip(self.sets[1:], outs)], "bf16")
        return st["gpu_launches"], [x[:k].clone() for (_, k), o in zip(res, outs) for x in o]


@pytest.mark.parametrize("order", ["batch first", "graph first"])
def test_first_call_of_each_is_tuned(order):
    torch = pytest.importorskip("torch")
    import mdet_gb300 as m

    # 10,000 contigs; a batch of 10,240 rows: the same logarithms
    calls = _Calls(torch, [_rows(10000, 1)] + [_rows(2048, 2 + k) for k in range(5)])
    first, second = (calls.batch, calls.graph) if order == "batch first" else (calls.graph, calls.batch)
    with m.Context(0) as alone, m.Context(0) as both:
        want, edges = second(alone)
        first(both)
        got, same = second(both)
    assert got == want
    assert all(torch.equal(a, b) for a, b in zip(edges, same))
