"""The ranks by 32-bit sorts where they can go wrong: scores that differ only
below the top 32 bits of their range, all equal, in runs of ties, crowded beyond
what is put in order in place (the full sort then), and few edges; and depths
whose variances are equal or below 1, with and without the correlation."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(ctx, fr, to, st, abd, var, **kw):
    ctx.set_abundance(abd, var)
    got = ctx.edges_sscr(fr, to, st, **kw)
    ctx.set_abundance(None, None)
    ref = oracle.sscr(fr, to, st, abd, var, **kw)
    assert np.allclose(got, ref, rtol=1e-12, atol=1e-12)


def _set(n, nabd, ne, seed):
    rng = np.random.default_rng(seed)
    abd = rng.lognormal(2.0, 0.8, (n, nabd)) + 1.01
    var = abd * rng.uniform(0.5, 2.0, (n, nabd))
    fr = rng.integers(0, n, ne)
    to = (fr + rng.integers(1, n, ne)) % n
    return rng, fr.astype(np.uint64), to.astype(np.uint64), abd, var


@pytest.mark.parametrize("ne", [1, 2, 255, 257, 20011])
@pytest.mark.parametrize("kind", ["spread", "equal", "ties", "crowded", "pairs"])
def test_scores(gpu_ctx, ne, kind):
    rng, fr, to, abd, var = _set(400, 4, ne, ne)
    if kind == "spread":
        st = rng.uniform(0.8, 1.0, ne)
    elif kind == "equal":
        st = np.full(ne, 0.93)
    elif kind == "ties":
        st = rng.choice([0.8, 0.9, 0.9 + 1e-16, 0.95, 1.0], ne)
    elif kind == "crowded":  # half the values within 2^-40 of the range
        st = np.where(rng.random(ne) < 0.5, 0.9 + rng.integers(0, 1000, ne) * 2.0 ** -52, rng.uniform(0.5, 1.0, ne))
    else:  # pairs that differ in the last bit
        st = np.repeat(rng.uniform(0.5, 1.0, (ne + 1) // 2), 2)[:ne]
        st[1::2] = np.nextafter(st[1::2], 0.0)
        st = rng.permutation(st)
    _check(gpu_ctx, fr, to, st, abd, var)


@pytest.mark.parametrize("nabd", [1, 2, 3, 11])
@pytest.mark.parametrize("min_cv", [0.0, 1e-7, 1.0])
def test_equal_and_small_variances(gpu_ctx, nabd, min_cv):
    rng, fr, to, abd, var = _set(300, nabd, 5000, 7 * nabd)
    var[:] = rng.choice([0.2, 0.9, 1.0, 3.0, 3.0005, 7.5], var.shape)
    abd[rng.random(abd.shape) < 0.05] = 5.0  # equal means too
    st = rng.uniform(0.8, 1.0, 5000)
    _check(gpu_ctx, fr, to, st, abd, var, min_cv=min_cv)
