"""How long label propagation's grid barriers wait (mdet_gb300/csrc/lp_wait.h): at
least the two seconds of every wait, at least a bound on what the slowest block
of a level may take, and no overflow at the largest sizes that the call accepts."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SPIN = 4000000000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("lp_wait")
    src = d / "w.cpp"
    src.write_text('#include "lp_wait.h"\n'
                   'extern "C" lpw::u64 level(lpw::u64 a, lpw::u64 b, lpw::u64 c, lpw::u64 d, lpw::u64 e)\n'
                   '{ return lpw::level_budget(a, b, c, d, e); }\n'
                   'extern "C" lpw::u64 sweep(lpw::u64 a, lpw::u64 b, lpw::u64 c, lpw::u64 d, lpw::u64 e, lpw::u64 f)\n'
                   '{ return lpw::sweep_budget(a, b, c, d, e, f); }\n')
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mdet_gb300", "csrc"), "-o",
                           str(d / "w.so"), str(src)])
    so = ctypes.CDLL(str(d / "w.so"))
    for f, k in ((so.level, 5), (so.sweep, 6)):
        f.restype = ctypes.c_uint64
        f.argtypes = [ctypes.c_uint64] * k
    return so


def test_grows_with_the_largest_contig(lib):
    # one contig of d edges over eight lanes: d / 8 rounds of at least four dependent
    # accesses at 1,000 cycles
    for d in (32, 1024, 100000, 4000000, 1 << 29):
        b = lib.level(1, 19456, 8, d, 2 * d)
        assert b >= SPIN + d // 8 * 4000
    assert lib.level(1, 19456, 8, 32, 64) < 1.01 * SPIN


@pytest.mark.parametrize("seed", range(5))
def test_covers_any_share(lib, seed):
    # contigs dealt to groups in turn, as the kernels do: the busiest group's rounds
    rng = np.random.default_rng(seed)
    groups, lanes = 64, 8
    deg = np.minimum((rng.pareto(1.0, 5000) * 3).astype(np.int64) + 1, 20000)
    rounds = [int((-(-deg[g::groups] // lanes)).sum()) for g in range(groups)]
    b = lib.level(deg.size, groups, lanes, int(deg.max()), int(deg.sum()))
    assert b >= SPIN + 4000 * max(rounds)
    s = lib.sweep(deg.size, groups, int(deg.max()), deg.size, 32 * groups, 32)
    assert s >= SPIN + 14000 * max(int(deg[g::groups].sum()) for g in range(groups))


def test_largest_sizes(lib):
    n, ne = 0x7FFFFFFE, 0x3FFFFFFE
    # not beyond what all the edges take, and far from 2^64
    assert SPIN < lib.level(n, 19456, 8, ne, 2 * ne) < 2 ** 42
    assert SPIN < lib.sweep(n, 608, 1024, n, 4864, 32) < 2 ** 47
