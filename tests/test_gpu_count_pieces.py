"""Counting with pieces sized by the whole: lengths around the smallest piece,
views that overlap so that the planned piece map does not hold them, set sizes
around the one-block plan, and a bad view among good ones."""
import numpy as np
import pytest

import mdet_gb300 as m
from oracle import oracle

pytestmark = pytest.mark.gpu


def _text(n, seed, width=61):
    rng = np.random.default_rng(seed)
    b = np.frombuffer(b"ACGTacgtN", np.uint8)[rng.choice(9, n, p=[.2, .2, .2, .2, .04, .04, .04, .04, .04])].copy()
    b[width - 1::width] = ord("\n")
    return b


def _check(ctx, data, off, ln):
    off, ln = np.asarray(off, np.uint64), np.asarray(ln, np.uint64)
    c, t = ctx.tnf_count(data, off, ln)
    oc, ot = oracle.tnf_count(data, off, ln)
    assert np.array_equal(c, oc)
    # float(c / rsum) against the rounded product with 1 / rsum: an ulp at a tie
    assert np.allclose(t, ot, rtol=2e-7, atol=0, equal_nan=True)


@pytest.mark.parametrize("width", [7, 61, 1 << 30])
def test_lengths_around_the_smallest_piece(gpu_ctx, width):
    lens = [0, 1, 3, 4, 5, 2047, 2048, 2049, 2051, 4095, 4096, 4100, 6143, 6145, 65535, 65536, 65537, 131073]
    data = _text(sum(lens) + len(lens), width % 1000, width)
    off = np.concatenate([[0], np.cumsum(np.array(lens) + 1)[:-1]])
    _check(gpu_ctx, data, off, lens)


@pytest.mark.parametrize("views", [3, 60, 700])
def test_overlapping_views(gpu_ctx, views):
    data = _text(90001, views)
    off = np.arange(views) * 7
    _check(gpu_ctx, data, off, data.size - off)


@pytest.mark.parametrize("n", [1, 1023, 1025, 8191, 8192, 8193])
def test_set_sizes_around_the_plan(gpu_ctx, n):
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 400, n)
    data = _text(int(lens.sum()) + 1, n)
    _check(gpu_ctx, data, np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)


def test_bad_view_then_good_call(gpu_ctx):
    data = _text(5000, 1)
    with pytest.raises(m.MdetError) as e:
        torch = pytest.importorskip("torch")
        d = torch.from_numpy(data).cuda()
        off = torch.tensor([0, 100, 4000], device="cuda")
        ln = torch.tensor([50, 100, 1001], device="cuda")
        out = torch.zeros(3 * 136, dtype=torch.int32, device="cuda")
        tnf = torch.zeros(3 * 136, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        gpu_ctx.tnf_count_dev(d.data_ptr(), 5000, off.data_ptr(), ln.data_ptr(), 3, out.data_ptr(), tnf.data_ptr())
    assert e.value.code == 1  # MDET_ERR_INVALID
    _check(gpu_ctx, data, [0, 2000], [2000, 3000])
