"""The record split's 64-byte newline counts at their edges: views that start,
end or lie whole inside one block, newline-only blocks, ragged file ends."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [0, 1, 15, 16, 63, 64, 65])
@pytest.mark.parametrize("width", [1, 3, 60, 63, 64, 1 << 20])
def test_views_around_blocks(gpu_ctx, tail, width):
    rng = np.random.default_rng(1000 * tail + width)
    out = []
    for k in range(260):
        seq = b"ACGT"[k % 4:k % 4 + 1] * int(rng.integers(0, 2 * k + 1))
        lines = [seq[i:i + width] for i in range(0, len(seq), width)]
        out.append(b">r%d%s\n" % (k, b" x>y" if k % 7 == 0 else b"") + b"\n".join(lines) + b"\n" * int(rng.integers(0, 3))
                   + b"\n")
    out.append(b">last\n" + b"\n" * 300 + b"A" * tail)
    data = np.frombuffer(b"".join(out), np.uint8)
    for min_contig in (0, 100):
        off, ln, sz, _, _, st = gpu_ctx.fasta_index(data, min_contig)
        so, sl, ssz, _, _ = oracle.fasta_index(data)
        keep = ssz >= min_contig
        assert st["n_records"] == so.size
        assert np.array_equal(off, so[keep]) and np.array_equal(ln, sl[keep]) and np.array_equal(sz, ssz[keep])


@pytest.mark.parametrize("rec", [b">a\n", b">b\nACGT\n", b">c x\n" + b"ACGTACGTAC\n" * 3])
def test_more_records_than_a_block_queues(gpu_ctx, rec):
    data = np.frombuffer(rec * (200000 // len(rec)) + b">tail\n" + b"A" * 3000, np.uint8)
    off, ln, sz, _, _, st = gpu_ctx.fasta_index(data, 0)
    so, sl, ssz, _, _ = oracle.fasta_index(data)
    assert st["n_records"] == so.size
    assert np.array_equal(off, so) and np.array_equal(ln, sl) and np.array_equal(sz, ssz)
