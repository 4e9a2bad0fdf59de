"""Recruiting by FP32 whole-bin means at bin sizes around a warp's members
and the runs of eight, with few and many samples (ties in the ranks at few):
the bins equal the oracle's, and widening the estimates' intervals, which
sends the pairs to the FP64 test, changes nothing."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nabd", [2, 3, 9, 17, 40])
def test_bin_sizes(gpu_ctx, nabd, monkeypatch):
    rng = np.random.default_rng(nabd)
    sizes_of = [10, 11, 31, 32, 33, 63, 64, 65, 256, 257, 300]
    label = np.repeat(np.arange(len(sizes_of)), sizes_of).astype(np.int64)
    prof = rng.lognormal(2, 1, (len(sizes_of), nabd))
    lone = rng.integers(0, len(sizes_of), 120)
    genome = np.concatenate([label, lone])
    label = np.concatenate([label, 1000 + np.arange(lone.size)])
    order = rng.permutation(label.size)
    label, genome = label[order], genome[order]
    abd = (prof[genome] * rng.lognormal(0, 0.3, (label.size, nabd))).astype(np.float32)
    sizes = np.where(label < 1000, 30000, 2600).astype(np.uint64)
    sg = rng.integers(0, len(sizes_of), 500)
    sabd = (prof[sg] * rng.lognormal(0, 0.3, (500, nabd))).astype(np.float32)
    ssz = rng.integers(1000, 2500, 500).astype(np.uint64)
    total = int(ssz.sum()) * 20
    want, swant, _ = oracle.recruit(abd, sabd, label, sizes, ssz, 200000, total)
    for scale in (None, "1e4", "1e7"):
        if scale:
            monkeypatch.setenv("MDET_RECRUIT_EPS_SCALE", scale)
        got, sgot, _ = gpu_ctx.recruit(abd, sabd, label, sizes, ssz, 200000, total)
        assert np.array_equal(got, want) and np.array_equal(sgot, swant)
