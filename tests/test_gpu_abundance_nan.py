"""Depths and variances that are not finite: the similarities of their edges are NaN and
sort above all others, so that they and the edges of the largest sTNF ranks score NaN
and no other does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [20, 5000])
@pytest.mark.parametrize("what", ["variance NaN", "variance inf", "depth NaN", "depth inf", "depth 1e200"])
def test_nan_similarities_rank_last(gpu_ctx, what, ne):
    rng = np.random.default_rng(ne)
    n = 2 * ne + 10
    abd = rng.lognormal(2.0, 0.8, (n, 1)) + 1.01
    var = abd * rng.uniform(0.5, 2.0, (n, 1))
    fr = np.arange(ne)
    bad = rng.permutation(ne - 4)[:2]  # their contigs are in no other edge
    value = {"NaN": np.nan, "inf": np.inf, "1e200": 1e200}[what.split()[1]]
    (var if what.startswith("variance") else abd)[bad] = value
    st = np.linspace(0.5, 0.9, ne)
    gpu_ctx.set_abundance(abd, var)
    got = gpu_ctx.edges_sscr(fr.astype(np.uint64), (fr + ne).astype(np.uint64), st, min_sample=5)
    gpu_ctx.set_abundance(None, None)
    assert set(np.flatnonzero(np.isnan(got)).tolist()) == {*bad.tolist(), ne - 2, ne - 1}
