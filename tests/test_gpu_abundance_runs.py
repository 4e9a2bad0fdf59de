"""Ranks of values that share their 32-bit keys: long runs of equal values (pairs
that saturate at the same similarity, one sTNF value for all), which are in order
as they stand, and runs with values out of order at the limit of what is put in
order in place (48)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _set(n, nabd, ne, seed):
    rng = np.random.default_rng(seed)
    abd = rng.lognormal(2.0, 0.8, (n, nabd)) + 1.01
    var = abd * rng.uniform(0.5, 2.0, (n, nabd))
    fr = rng.integers(0, n, ne)
    to = (fr + rng.integers(1, n, ne)) % n
    return rng, fr.astype(np.uint64), to.astype(np.uint64), abd, var


def _scores(ctx, fr, to, st, abd, var, **kw):
    ctx.set_abundance(abd, var)
    ctx.edges_sscr(fr, to, st, **kw)  # buffers and modules in place
    ctx.set_timing(True)
    try:
        got = ctx.edges_sscr(fr, to, st, **kw)
        ms = ctx.kernel_ms("abd_ranks")[0]
    finally:
        ctx.set_timing(False)
        ctx.set_abundance(None, None)
    ref = oracle.sscr(fr, to, st, abd, var, **kw)
    # the accuracy that the header states
    assert np.allclose(got, ref, rtol=1e-12, atol=1e-12)
    return ms


@pytest.mark.parametrize("kind", ["saturated", "equal"])
def test_long_runs_take_no_serial_walk(gpu_ctx, kind):
    # 500,000 dependent gathers by one thread take 50 ms at the 100 ns of an L2
    # hit; the passes over 500,000 values take well under 1 ms
    rng, fr, to, abd, var = _set(2000, 1, 500000, 3)
    st = rng.uniform(0.5, 1.0, fr.size)
    if kind == "saturated":  # even and odd contigs far apart: one similarity for all edges
        abd[::2] += 5000.0
        fr, to = fr // 2 * 2, to // 2 * 2 + 1
    else:
        st[:] = 0.93
    assert _scores(gpu_ctx, fr, to, st, abd, var) < 10.0


@pytest.mark.parametrize("run", [2, 47, 48, 49, 50, 97])
@pytest.mark.parametrize("place", ["front", "middle", "end"])
def test_runs_at_the_limit(gpu_ctx, run, place):
    rng, fr, to, abd, var = _set(400, 4, 6000, run)
    st = rng.uniform(0.5, 1.0, fr.size)
    st[:2] = 0.5, np.nextafter(1.0, 0.0)  # the range, whatever the draw
    base = {"front": 0.5, "middle": 0.75, "end": np.nextafter(1.0, 0.0) - 256 * 2.0 ** -53}[place]
    at = rng.permutation(np.arange(2, fr.size))[:run]
    st[at] = base + rng.permutation(run) * 2.0 ** -53
    st[at[:2]] = st[at[0]]  # and a tie
    _scores(gpu_ctx, fr, to, st, abd, var)
