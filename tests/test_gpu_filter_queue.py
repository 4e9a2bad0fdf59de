"""The tensor-core filter's hit queues: genomes whose contigs lie side by side in
the prepared order, of sizes that give a warp's 32 x 64 chunk every number of
hits from a few to hundreds -- below, at and above the half queue (16, 32 or 128
hits by tile shape) at which a warp flushes or writes to the list itself.  The
pairs above the cutoff are the plain form's, whatever the shape, call after call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _genomes(sizes, seed):
    rng = np.random.default_rng(seed)
    g = np.repeat(np.arange(len(sizes)), sizes)
    c = rng.dirichlet(np.full(136, 0.4), len(sizes))[g] * 4000.0 + rng.uniform(0, 4, (g.size, 136))
    tnf = (c / np.sqrt((c * c).sum(1, keepdims=True))).astype(np.float32)
    return tnf, np.log10(20000.0 + 20.0 * np.arange(g.size))


@pytest.mark.parametrize("sizes", [list(range(1, 49)), [5, 6] * 200, [8] * 150 + [1] * 300, [17, 33, 65, 129] * 8],
                         ids=["1-48", "pairs", "mixed", "tile edges"])
def test_hits_per_chunk(gpu_ctx, sizes):
    torch = pytest.importorskip("torch")
    tnf, ls = _genomes(sizes, len(sizes))
    n, me = ls.size, 200
    d_tnf, d_ls = torch.from_numpy(tnf).cuda(), torch.from_numpy(ls).cuda()

    def edges(mode):
        fr, to = (torch.zeros(n * me, dtype=torch.int64, device="cuda") for _ in range(2))
        st = torch.zeros(n * me, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        k, stats = gpu_ctx.tnf_graph_dev(d_tnf.data_ptr(), d_ls.data_ptr(), n, 0.9, me, mode, fr.data_ptr(),
                                         to.data_ptr(), st.data_ptr(), n * me)
        return k, stats["n_above_cutoff"], fr, to, st

    ref = edges("plain")
    assert ref[1] >= sum(s * (s - 1) // 2 for s in sizes)
    try:
        for shape in (128256, 128128, 256128):
            gpu_ctx.set_autotune(shape)
            for mode in ("bf16", "tf32"):
                for _ in range(5):
                    got = edges(mode)
                    assert got[:2] == ref[:2]
                    assert all(torch.equal(a, b) for a, b in zip(got[2:], ref[2:]))
    finally:
        gpu_ctx.set_autotune(1)
