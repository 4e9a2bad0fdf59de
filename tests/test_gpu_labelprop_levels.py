"""Label propagation with many levels and with contigs at the edges of the
warp and block forms: a path (one level per contig), rings of cliques with 31
to 34 edges a contig, a hub next to a path, and stretches longer than the first
traversal pass; bins and sweeps as the oracle's."""
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


def test_path_of_levels(gpu_ctx):
    n = 2600
    i = np.arange(n - 1)
    st = _check(gpu_ctx, i, i + 1, 0.999 - 1e-5 * i, n)
    assert st["levels_max"] > 1000


@pytest.mark.parametrize("size", [32, 33, 34, 35])
def test_cliques_around_a_warp(gpu_ctx, size):
    rng = np.random.default_rng(size)
    k = 40
    a, b = np.triu_indices(size, 1)
    fr = np.concatenate([a + c * size for c in range(k)] + [np.arange(k) * size])
    to = np.concatenate([b + c * size for c in range(k)] + [(np.arange(k) * size + size) % (k * size)])
    sc = rng.uniform(0.62, 0.99, fr.size)
    _check(gpu_ctx, fr, to, sc, k * size)


def test_hub_beside_a_path(gpu_ctx):
    rng = np.random.default_rng(3)
    n = 5000
    spokes = np.arange(1, 2300)
    i = np.arange(2300, n - 1)
    fr = np.concatenate([np.zeros(spokes.size, int), i, rng.integers(0, n, 4000)])
    to = np.concatenate([spokes, i + 1, rng.integers(0, n, 4000)])
    ok = fr != to
    sc = rng.uniform(0.5, 1.0, fr.size)
    _check(gpu_ctx, np.minimum(fr, to)[ok], np.maximum(fr, to)[ok], sc[ok], n)


def test_stretches_over_several_passes(gpu_ctx):
    rng = np.random.default_rng(4)
    n, ne = 3000, 400000  # six passes of growing size
    g = rng.integers(0, 12, n)
    a, b = rng.integers(0, n, ne), rng.integers(0, n, ne)
    # most of the best-scored edges join few contigs, so late stretches are long
    a[: ne // 2], b[: ne // 2] = a[: ne // 2] % 300, b[: ne // 2] % 300
    sc = np.where(g[a] == g[b], 0.7 + 0.3 * rng.random(ne), 0.4 + 0.3 * rng.random(ne))
    sc[: ne // 2] = 0.95 + 0.05 * rng.random(ne // 2)
    ok = a != b
    _check(gpu_ctx, a[ok], b[ok], sc[ok], n)
