"""The record split of files with millions of short records, as raw assemblies have
them: one scan for records from 200 bytes on at any file size, and the same records
as the layout says; records too dense for the queues take the second scan."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("records,length,scans", [(4300000, 280, 1), (6000000, 200, 1), (1000000, 700, 1),
                                                  (900000, 90, 1), (8000000, 50, 2), (3000, 5, 2)])
def test_repeated_record(gpu_ctx, records, length, scans):
    # a queue holds 2,304 starts; a block's range is 384 KB at most, and smaller where
    # sixteen blocks an SM make it so (33 KB at 900,000 x 90 bytes, 164 KB at 8,000,000 x 50)
    torch = pytest.importorskip("torch")
    head = b">contig_x len\n" if length > 20 else b">a\n"
    rec = head + b"ACGTACGTAC" * ((length - len(head) - 1) // 10 + 1)
    rec = rec[:length - 1] + b"\n"
    buf = torch.tensor(list(rec), dtype=torch.uint8, device="cuda").repeat(records)
    n = buf.numel()
    buf = torch.cat([buf, torch.zeros(64, dtype=torch.uint8, device="cuda")])
    off, ln, size, noff = (torch.zeros(records, dtype=torch.int64, device="cuda") for _ in range(4))
    ls = torch.zeros(records, dtype=torch.float64, device="cuda")
    nlen = torch.zeros(records, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.set_timing(True)
    try:
        st = gpu_ctx.fasta_index_dev(buf.data_ptr(), n, 1, records, off.data_ptr(), ln.data_ptr(), size.data_ptr(),
                                     ls.data_ptr(), noff.data_ptr(), nlen.data_ptr())
        passes = sum(gpu_ctx.kernel_ms(k)[1] for k in ("k_fa_scan", "k_fa_scan_append"))
    finally:
        gpu_ctx.set_timing(False)
    assert passes == scans
    assert st["n_records"] == st["n_large"] == records
    start = torch.arange(records, device="cuda") * length
    assert torch.equal(off, start + len(head)) and torch.equal(noff, start + 1)
    seq = length - len(head) - 1
    assert torch.all(ln == seq) and torch.all(size == seq) and torch.all(nlen == (8 if length > 20 else 1))
