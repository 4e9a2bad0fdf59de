"""Views that overlap are counted in pieces sized by what they hold together: as fast
as the same bytes side by side, and the same counts, below and above the contigs that
one block plans."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,length", [(3, 60000), (900, 70001), (8192, 2500), (8193, 2500), (9000, 9001)])
def test_counts(gpu_ctx, n, length):
    rng = np.random.default_rng(n)
    data = np.frombuffer(b"ACGTNacgt\n", np.uint8)[rng.integers(0, 10, 80000)]
    off = rng.integers(0, data.size - length + 1, n).astype(np.uint64)
    ln = np.full(n, length, np.uint64)
    c, _ = gpu_ctx.tnf_count(data, off, ln)
    oc, _ = oracle.tnf_count(data, off, ln)
    assert np.array_equal(c, oc)


def test_time_of_overlapping_views(gpu_ctx):
    torch = pytest.importorskip("torch")
    n, length = 800, 2500000  # 2 GB in all
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    one = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[
        torch.randint(0, 4, (length + 64,), generator=gen, device="cuda")]
    wide = torch.cat([one[:length].repeat(n), one[:64]])
    counts = torch.empty(n, 136, dtype=torch.int32, device="cuda")
    tnf = torch.empty(n, 136, dtype=torch.float32, device="cuda")
    ln = torch.full((n,), length, dtype=torch.int64, device="cuda")
    ms, got = {}, {}
    for name, buf, off in (("side", wide, torch.arange(n, device="cuda") * length), ("over", one, torch.zeros_like(ln))):
        torch.cuda.synchronize()
        times = []
        for _ in range(5):
            gpu_ctx.set_timing(True)
            gpu_ctx.tnf_count_dev(buf.data_ptr(), buf.numel() - 64, off.data_ptr(), ln.data_ptr(), n, counts.data_ptr(),
                                  tnf.data_ptr())
            times.append(gpu_ctx.kernel_ms("k_count")[0])
            gpu_ctx.set_timing(False)
        ms[name], got[name] = sorted(times)[2], counts.clone()
    assert torch.equal(got["side"], got["over"])
    # the same work, from L2 instead of memory; pieces of 2 KB take 1.6 times as long
    assert ms["over"] < 1.25 * ms["side"]
