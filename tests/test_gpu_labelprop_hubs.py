"""Label propagation with contigs of more edges than a group or a block sorts in shared memory
(1,024; 2,048), which are swept by a launch per level: degrees around those limits, hubs with
exact ties and with distinct scores, among chains and cliques."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(ctx, fr, to, sc, n, **kw):
    fr, to, sc = np.asarray(fr, np.uint64), np.asarray(to, np.uint64), np.asarray(sc, np.float64)
    mem, st = ctx.label_propagation(fr, to, sc, n, **kw)
    omem, ost = oracle.label_prop(fr, to, sc, n, **kw)
    assert np.array_equal(mem, omem)
    return st


@pytest.mark.parametrize("degree", [1022, 1023, 1024, 1025, 2047, 2048, 2049, 2300, 40000])
@pytest.mark.parametrize("scores", ["distinct", "ties"])
def test_hub_among_cliques(gpu_ctx, degree, scores):
    rng = np.random.default_rng(degree)
    spokes = np.arange(1, degree + 1)
    a, b = np.triu_indices(34, 1)
    base = degree + 1 + 34 * np.arange(20)
    fr = np.concatenate([np.zeros(degree, int)] + [a + k for k in base] + [np.arange(degree + 1, degree + 600)])
    to = np.concatenate([spokes] + [b + k for k in base] + [np.arange(degree + 2, degree + 601)])
    n = degree + 1 + 34 * 20
    sc = rng.uniform(0.62, 0.99, fr.size)
    if scores == "ties":
        sc[:degree] = 0.875
    ok = rng.permutation(fr.size)
    st = _check(gpu_ctx, fr[ok], to[ok], sc[ok], n)
    assert st["degree_max"] >= degree * 9 // 10  # the last run may end before the last spoke


def test_many_hubs(gpu_ctx):
    rng = np.random.default_rng(1)
    n, hubs = 30000, 12
    fr = np.concatenate([rng.integers(0, hubs, 40000), rng.integers(0, n, 30000)])
    to = np.concatenate([rng.integers(hubs, n, 40000), rng.integers(0, n, 30000)])
    ok = fr != to
    key = np.unique(np.minimum(fr, to)[ok] * n + np.maximum(fr, to)[ok])
    sc = rng.uniform(0.55, 1.0, key.size)
    st = _check(gpu_ctx, key // n, key % n, sc, n)
    assert st["degree_max"] > 1024


def test_large_hub(gpu_ctx):
    # a star whose hub takes a few tenths of a second a sweep
    rng = np.random.default_rng(2)
    n = 250001
    st = _check(gpu_ctx, np.zeros(n - 1, int), 1 + rng.permutation(n - 1), rng.uniform(0.62, 0.99, n - 1), n)
    assert st["degree_max"] > 200000
