"""Counts at the sizes where the pieces change: buffers around 4 MB (pieces of 4 and
8 KB), contigs around a piece, and maps around what the one-block plan fills."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(ctx, lens, seed):
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens, np.uint64)
    off = np.concatenate([[0], np.cumsum(lens + 1)[:-1]]).astype(np.uint64)
    data = np.frombuffer(b"ACGTacgtN\n", np.uint8)[rng.integers(0, 10, int(lens.sum()) + lens.size)]
    c, _ = ctx.tnf_count(data, off, lens)
    oc, _ = oracle.tnf_count(data, off, lens)
    assert np.array_equal(c, oc)


@pytest.mark.parametrize("total", [(4 << 20) - 40000, 4 << 20, (4 << 20) + 40000])
def test_around_four_megabytes(gpu_ctx, total):
    lens = np.array([4095, 4096, 4097, 8191, 8192, 8193, 12289] * 100)
    lens = lens[np.cumsum(lens + 1) < total]
    _check(gpu_ctx, np.append(lens, total - lens.sum() - lens.size - 1), total)


@pytest.mark.parametrize("n", [8192, 8193])
def test_around_the_plan(gpu_ctx, n):
    # pieces of 8 KB, three or four to a contig: maps of 56,000 and 68,000 entries
    for length in (24000, 30000):
        _check(gpu_ctx, np.full(n, length) + np.arange(n) % 7, length + n)
