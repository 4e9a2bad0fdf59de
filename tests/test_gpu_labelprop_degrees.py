"""Levels of contigs whose degrees lie around what a warp or eight lanes take at a
time (8, 32, 33, 128 neighbours and remainders), many of them in one level and one
after another; bins and sweeps as the oracle's."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(ctx, fr, to, sc, n):
    fr, to, sc = np.asarray(fr, np.uint64), np.asarray(to, np.uint64), np.asarray(sc, np.float64)
    mem, st = ctx.label_propagation(fr, to, sc, n)
    omem, ost = oracle.label_prop(fr, to, sc, n)
    assert np.array_equal(mem, omem)
    assert st["sweeps"] == ost["sweeps"]


@pytest.mark.parametrize("degree", [7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 257])
def test_stars(gpu_ctx, degree):
    # 40 stars in a ring, their spokes scored above the ring
    rng = np.random.default_rng(degree)
    k, per = 40, degree - 1  # a hub has its spokes and two ring edges, less the one that closes
    hub = np.arange(k) * (per + 1)
    fr = np.concatenate([np.repeat(hub, per), hub])
    to = np.concatenate([(hub[:, None] + 1 + np.arange(per)).ravel(), np.roll(hub, -1)])
    sc = np.concatenate([rng.uniform(0.8, 0.99, k * per), rng.uniform(0.62, 0.7, k)])
    _check(gpu_ctx, fr, to, sc, k * (per + 1))


@pytest.mark.parametrize("n,deg", [(400, 30), (700, 130), (3000, 60)])
def test_random_degrees(gpu_ctx, n, deg):
    rng = np.random.default_rng(n)
    w = rng.pareto(1.5, n) + 0.2
    a, b = (rng.choice(n, n * deg, p=w / w.sum()) for _ in range(2))
    ok = a != b
    key = np.unique(np.minimum(a, b)[ok] * n + np.maximum(a, b)[ok])
    _check(gpu_ctx, key // n, key % n, rng.uniform(0.55, 1.0, key.size), n)
