"""Stretches of the traversal whose lengths change: a long one after short ones (most
of its edges join contigs of one bin), short ones after a long one, and an end
within a pass that the stretch before it made long; bins as the oracle's."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long_at", [0.1, 0.5, 0.9])
@pytest.mark.parametrize("low", [0.0, 0.2])
def test_long_and_short_stretches(gpu_ctx, long_at, low):
    rng = np.random.default_rng(int(100 * long_at))
    n, size = 4000, 20
    g = np.arange(n) // size
    # every group's edges at its own score, group after group; at `long_at` 600,000 more
    # edges among the contigs of the groups before
    a = np.repeat(np.arange(n), 6)
    b = g[a] * size + rng.integers(0, size, a.size)
    sc = 0.98 - 0.3 * (g[a] + rng.random(a.size)) / (n // size)
    before = int(long_at * n)
    c = rng.integers(0, before, 600000)
    d = g[c] * size + rng.integers(0, size, c.size)
    mid = 0.98 - 0.3 * long_at
    fr, to = np.concatenate([a, c]), np.concatenate([b, d])
    sc = np.concatenate([sc, mid - 1e-4 * rng.random(c.size)])
    last = rng.random(sc.size) < low  # below min_s: the traversal's early end
    sc = np.where(last, 0.1 + 0.5 * rng.random(sc.size), sc)
    ok = fr != to
    fr, to, sc = fr[ok].astype(np.uint64), to[ok].astype(np.uint64), sc[ok]
    mem, st = gpu_ctx.label_propagation(fr, to, sc, n)
    omem, ost = oracle.label_prop(fr, to, sc, n)
    assert np.array_equal(mem, omem)
    assert all(st[k] == ost[k] for k in ("calls", "sweeps", "graph_edges", "connected"))
