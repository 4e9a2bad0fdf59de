"""The 32-bit keys of the ranks spread what scoring meets: genomes whose contigs
correlate closely, few and many samples, contigs of constant depth (whose
correlations are NaN).  None of these falls back to the full sort, and the scores
are the oracle's; correlations of +-1 but for their last bits too."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _set(n, nabd, deg, seed):
    """Depths and edges of an assembly: 85 % of the edges within a genome."""
    rng = np.random.default_rng(seed)
    genomes = max(3, n // 450)
    genome = rng.integers(0, genomes, n)
    depth = np.exp(rng.normal(size=(genomes, nabd)) + np.log(10.0))
    abd = (depth[genome] * np.exp(0.15 * rng.normal(size=(n, nabd)))).astype(np.float32).astype(np.float64) + 1.01
    var = abd * rng.uniform(0.5, 2.0, abd.shape)
    order = np.argsort(genome, kind="stable")
    count = np.bincount(genome, minlength=genomes)
    first = count.cumsum() - count
    fr = rng.integers(0, n, int(0.8 * n * deg))
    mate = order[first[genome[fr]] + (rng.random(fr.size) * count[genome[fr]]).astype(np.int64)]
    to = np.where(rng.random(fr.size) < 0.85, mate, rng.integers(0, n, fr.size))
    ok = fr != to
    fr, to = fr[ok], to[ok]
    v = rng.random(fr.size)
    st = np.where(genome[fr] == genome[to], 1 - 0.35 * v ** 1.5, 0.9 - 0.5 * np.sqrt(v))
    return fr.astype(np.uint64), to.astype(np.uint64), st, abd, var


def _run(ctx, fr, to, st, abd, var, **kw):
    ctx.set_abundance(abd, var)
    ctx.set_timing(True)
    try:
        got = ctx.edges_sscr(fr, to, st, **kw)
        passes = [ctx.kernel_ms(k)[1] for k in ("abd_ranks", "abd_ranks_full")]
    finally:
        ctx.set_timing(False)
        ctx.set_abundance(None, None)
    return got, passes


@pytest.mark.parametrize("n,nabd,deg", [(60000, 10, 80), (60000, 6, 80), (60000, 4, 80), (60000, 3, 80),
                                        (60000, 1, 80), (90000, 3, 100), (90000, 16, 100), (1501, 3, 21)])
def test_no_fallback(gpu_ctx, n, nabd, deg):
    fr, to, st, abd, var = _set(n, nabd, deg, nabd)
    got, passes = _run(gpu_ctx, fr, to, st, abd, var)
    assert passes == [1, 0]
    # the accuracy that the header states
    assert np.allclose(got, oracle.sscr(fr, to, st, abd, var), rtol=1e-12, atol=1e-12)


def test_contigs_of_constant_depth(gpu_ctx):
    fr, to, st, abd, var = _set(60000, 10, 80, 5)
    abd[::1000] = 12.0
    got, passes = _run(gpu_ctx, fr, to, st, abd, var)
    assert passes == [1, 0] and np.isfinite(got).all()


@pytest.mark.parametrize("nabd,ne", [(2, 30011), (3, 30011), (5, 257)])
def test_correlations_at_the_ends(gpu_ctx, nabd, ne):
    # depths on two lines, rising and falling: every correlation is 1 or -1, give
    # or take the last bits
    rng = np.random.default_rng(ne)
    n = 1000
    line = 10.0 + 3.0 * np.arange(nabd)
    abd = np.where(rng.random((n, 1)) < 0.5, line, line[::-1]) * rng.uniform(0.5, 2.0, (n, 1))
    var = abd * rng.uniform(0.5, 2.0, abd.shape)
    fr = rng.integers(0, n, ne)
    to = (fr + rng.integers(1, n, ne)) % n
    st = rng.uniform(0.8, 1.0, ne)
    fr, to = fr.astype(np.uint64), to.astype(np.uint64)
    got, _ = _run(gpu_ctx, fr, to, st, abd, var, min_sample=2)
    assert np.allclose(got, oracle.sscr(fr, to, st, abd, var, min_sample=2), rtol=1e-12, atol=1e-12)
