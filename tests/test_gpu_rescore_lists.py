"""The re-scoring lane's lists: per level the columns to evaluate, and the factors among
them, whose sums of squares the QR starts from (a shared column's are read by nobody)."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SRC = Path(__file__).resolve().parent / "native" / "rescore_harness.cu"
EVAL, COPY, WHOLE, STOP, SHARED = 1, 2, 0, 1, 2


@pytest.fixture(scope="module")
def lists(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = tmp_path_factory.mktemp("rescore") / "rescore.so"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-shared", "-Xcompiler", "-fPIC", str(SRC), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.rescore_levels.argtypes = [C.c_void_p] * 3 + [C.c_int32] + [C.c_void_p] * 4

    def run(need, kind, level_end):
        need, kind = np.ascontiguousarray(need, np.uint8), np.ascontiguousarray(kind, np.uint8)
        level_end = np.ascontiguousarray(level_end, np.int32)
        cols, fac = np.full(len(need), -7, np.int32), np.full(len(need), -7, np.int32)
        count, fac_count = np.zeros(len(level_end), np.int32), np.zeros(1, np.int32)
        assert lib.rescore_levels(need.ctypes.data, kind.ctypes.data, level_end.ctypes.data, len(level_end),
                                  cols.ctypes.data, count.ctypes.data, fac.ctypes.data, fac_count.ctypes.data) == 0
        return cols, count, fac, int(fac_count[0])
    return run


@pytest.mark.parametrize("sizes", [[1], [31, 1], [1024], [1025, 0, 3], [2500, 700, 1024, 1]])
@pytest.mark.parametrize("share", [0.0, 0.4, 1.0])
def test_lists(lists, sizes, share):
    rng = np.random.default_rng(len(sizes) * 10 + int(share * 5))
    end = np.cumsum(sizes)
    n = int(end[-1])
    need = rng.choice([0, EVAL, COPY], n)
    kind = np.where(rng.random(n) < share, SHARED, rng.choice([WHOLE, STOP], n))
    cols, count, fac, n_fac = lists(need, kind, end)
    for lo, hi, k in zip(np.r_[0, end[:-1]], end, count):
        want = lo + np.flatnonzero(need[lo:hi] == EVAL)
        assert k == len(want) and np.array_equal(cols[lo:lo + k], want)
    want = np.flatnonzero((need == EVAL) & (kind != SHARED))
    assert n_fac == len(want) and np.array_equal(fac[:n_fac], want) and np.all(fac[n_fac:] == -1)
