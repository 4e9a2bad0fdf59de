"""The training gradient at batch sizes around the edges of its kernels: one
128-row tile with one real pair, a tile boundary and one past it, spans of
several 64-row chunks, and more row tiles than one per SM."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))

from oracle import mlp_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npairs", [1, 64, 65, 700, 4999, 10100])
def test_gradient_sizes(gpu_ctx, npairs):
    import mdet_gb300 as m

    rng = np.random.default_rng(npairs)
    rows = min(2 * npairs, 3001)
    x = rng.normal(0.0, 0.08, (rows, R.IN)).astype(np.float32) + 0.05
    pairs = rng.integers(0, rows, (npairs, 2)).astype(np.uint32)
    pairs[:, 1] = np.where(pairs[:, 0] == pairs[:, 1], (pairs[:, 1] + 1) % rows, pairs[:, 1])
    y = (rng.random(npairs) < 0.5).astype(np.float32)
    net = m.Network(gpu_ctx, seed=3)
    p = net.get_params()
    e = np.linalg.norm(R.embed(p, x[pairs[:, 0]]) - R.embed(p, x[pairs[:, 1]]), axis=1)
    mp, mn = 0.7 * float(np.median(e)), 1.3 * float(np.median(e))
    loss, g = net.grad(x, pairs, y, mp, mn)
    net.close()
    rl, rg = R.loss_and_grad_bf16(p, x, pairs, y, mp, mn)
    assert abs(loss - rl) <= 1e-4 * abs(rl) + 1e-9
    # a GEMM operand on the other side of a BF16 rounding boundary moves by
    # 2^-8 of itself, a product of two by 2^-7; accumulation is FP32
    for lo, hi in [(R.W1, R.B1), (R.B1, R.W2), (R.W2, R.B2), (R.B2, R.W3), (R.W3, R.B3)]:
        err = np.linalg.norm(g[lo:hi] - rg[lo:hi]) / max(np.linalg.norm(rg[lo:hi]), 1e-30)
        assert err < 2.0 ** -7, (lo, hi, err)
