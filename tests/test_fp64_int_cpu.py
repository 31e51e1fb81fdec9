"""FP64 operations formed on the integer pipes (csrc/common/fp64_int.h) and the
split elementary functions (csrc/common/rr_math_split.h) on the host: the same
bits as the native operations and as rr_math.h, over random significands,
operands next to half-way points and the special values (CPU only)."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
OPS = ["mul", "div", "sqrt", "lt", "eq", "sin", "cos", "log", "exp", "mul_by", "scaled", "scaled2"]
SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, 0.5, 2.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                    2.225073858507201e-308, 1.7976931348623157e308, -1.7976931348623157e308, 3.0, 1.0 + 2.0**-52,
                    1.0 - 2.0**-53, 2.0 - 2.0**-52, 0.7853981633974483, np.nextafter(0.7853981633974483, 1), 1048576.0,
                    np.nextafter(1048576.0, 0), 708.0, 709.782712893384, 709.7827128933841, -745.1332191019412,
                    -745.1332191019411, 1e-160, 1e160, 1.4142135623730951, 1.414213562373095])


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    gcc = shutil.which("gcc")
    if not gcc:
        pytest.skip("gcc not available")
    so = tmp_path_factory.mktemp("fi") / "fp64_int_harness.so"
    subprocess.run([gcc, "-std=c99", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                    str(HERE / "native" / "fp64_int_harness.c"), "-o", str(so), "-lm"], check=True)
    lib = C.CDLL(str(so))
    lib.fi_apply.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p]

    def run(op, a, b):
        a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b))
        out = np.empty((2, len(a)))
        for native in (0, 1):
            lib.fi_apply(OPS.index(op), native, a.ctypes.data, b.ctypes.data, len(a), out[native].ctypes.data)
        return out
    return run


def operands(op, seed, n=400_000):
    rng = np.random.default_rng(seed)
    bits = rng.integers(0, 2**52, n, dtype=np.uint64)
    near = rng.random(n) < 0.3  # significands of few bits: products and quotients next to ties
    bits[near] &= np.uint64(0xfffff00000000000)
    exps = rng.integers(1023 - 40, 1023 + 40, n).astype(np.uint64)
    wide = rng.random(n) < 0.1
    exps[wide] = rng.integers(0, 2048, int(wide.sum())).astype(np.uint64)
    sign = rng.integers(0, 2, n).astype(np.uint64)
    a = (bits | exps << np.uint64(52) | sign << np.uint64(63)).view(np.float64)
    b = a[rng.permutation(n)].copy()
    with np.errstate(all="ignore"):
        if op == "div":  # a a rounded multiple of b: quotients next to representable values and half-way points
            half = rng.random(n) < 0.4
            q = np.nextafter(1.0 + rng.integers(0, 2**20, n) * 2.0**-20, rng.choice([0.0, 4.0], n))
            a[half] = (b * q)[half]
        if op == "sqrt":
            sq = rng.random(n) < 0.4
            a = np.abs(a)
            a[sq] = np.nextafter(a[sq] * a[sq], rng.choice([0.0, np.inf], int(sq.sum())))
        if op in ("eq", "lt"):
            same = rng.random(n) < 0.3
            b[same] = a[same]
    s = np.array([(x, y) for x in SPECIAL for y in SPECIAL]).T
    return np.concatenate([a, s[0], rng.choice(SPECIAL, 2000)]), np.concatenate([b, s[1], b[:2000]])


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_same_bits(apply, op, seed):
    a, b = operands(op, seed)
    if op in ("sin", "cos"):
        a = np.concatenate([a, np.random.default_rng(seed).uniform(-20, 20, 200_000),
                            np.arange(-4000, 4000) * (np.pi / 4)])
    if op in ("log", "exp"):
        a = np.concatenate([a, np.random.default_rng(seed).uniform(0, 50, 200_000),
                            np.random.default_rng(seed).uniform(-745, 710, 100_000)])
    got, ref = apply(op, a, np.resize(b, len(a)))
    same = (got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), (op, a[~same][:3], np.resize(b, len(a))[~same][:3], got[~same][:3], ref[~same][:3])
