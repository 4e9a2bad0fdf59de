"""Label propagation whose levels are wide in contigs of more than 32 edges: cliques
that are traversed one after another, so that a run's levels hold one contig of
every clique so far -- past the width at which sweeps go by a launch per level, and
cliques of 33 and fewer besides, whose contigs take a warp."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cliques,size,small", [(420, 40, 0), (300, 66, 200), (100, 130, 900), (230, 34, 33)])
def test_levels_of_cliques(gpu_ctx, cliques, size, small):
    rng = np.random.default_rng(cliques)
    fr, to, sc, n = [], [], [], 0
    for k in range(cliques + small):
        s = size if k % (1 + small // cliques) == 0 and k < cliques * (1 + small // cliques) else 12 + k % 22
        a, b = np.triu_indices(s, 1)
        fr.append(a + n)
        to.append(b + n)
        sc.append(0.99 - 0.3 * (k + rng.random(a.size)) / (cliques + small))
        n += s
    fr, to, sc = (np.concatenate(x) for x in (fr, to, sc))
    mem, st = gpu_ctx.label_propagation(fr.astype(np.uint64), to.astype(np.uint64), sc, n)
    omem, ost = oracle.label_prop(fr.astype(np.uint64), to.astype(np.uint64), sc, n)
    assert np.array_equal(mem, omem)
    assert st["sweeps"] == ost["sweeps"] and st["ties"] == ost["ties"]
