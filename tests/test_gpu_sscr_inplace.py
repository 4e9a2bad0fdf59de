"""Scores written over the sTNF values they are made from, with values that the
32-bit ranks cannot order (the full sort follows) and with values that they can."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _edges(n, nabd, ne, seed):
    rng = np.random.default_rng(seed)
    genome = rng.integers(0, max(3, n // 450), n)
    depth = np.exp(rng.normal(size=(genome.max() + 1, nabd)) + np.log(10.0))
    abd = depth[genome] * np.exp(0.15 * rng.normal(size=(n, nabd))) + 1.01
    var = abd * rng.uniform(0.5, 2.0, abd.shape)
    fr = rng.integers(0, n, ne)
    to = (fr + rng.integers(1, n, ne)) % n
    return rng, fr, to, abd, var


@pytest.mark.parametrize("values", ["spread", "crowded"])
@pytest.mark.parametrize("nabd,ne", [(3, 260000), (2, 20011), (4, 20011), (10, 20011)])
def test_in_place(gpu_ctx, nabd, ne, values):
    torch = pytest.importorskip("torch")
    rng, fr, to, abd, var = _edges(3000, nabd, ne, nabd)
    st = rng.uniform(0.5, 1.0, ne)
    if values == "crowded":  # half of them within 1,000 steps of 2^-52 of one another
        st = np.where(rng.random(ne) < 0.5, 0.9 + rng.integers(0, 1000, ne) * 2.0 ** -52, st)
    f, t, src = (torch.from_numpy(x).cuda() for x in (fr, to, st))
    out, same = torch.empty_like(src), src.clone()
    gpu_ctx.set_abundance(abd, var)
    torch.cuda.synchronize()
    gpu_ctx.edges_sscr_dev(f.data_ptr(), t.data_ptr(), src.data_ptr(), ne, out.data_ptr(), min_sample=2)
    gpu_ctx.edges_sscr_dev(f.data_ptr(), t.data_ptr(), same.data_ptr(), ne, same.data_ptr(), min_sample=2)
    torch.cuda.synchronize()
    gpu_ctx.set_abundance(None, None)
    assert torch.equal(same, out) and torch.equal(src, torch.from_numpy(st).cuda())
    ref = oracle.sscr(fr.astype(np.uint64), to.astype(np.uint64), st, abd, var, min_sample=2)
    # the accuracy that the header states
    assert np.allclose(out.cpu().numpy(), ref, rtol=1e-12, atol=1e-12)
