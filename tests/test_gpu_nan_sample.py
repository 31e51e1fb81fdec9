"""The certificate for candidates with a NaN column beyond the first one, which
looks at 2048 sampled rows before it looks at all: columns that differ from one
another, or from zero, only on rows outside the sample or only inside it, exact
duplicates, and well-conditioned ones, on both sides of the one-launch form's
32768 rows: the oracle's bits."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import CERTIFIED, PLAIN, Context, encode

pytestmark = pytest.mark.gpu
TREES = ["add x0 add x1 ln x2", "add x0 add x3 ln x2", "add x0 add x4 ln x2", "add x0 add x5 ln x2",
         "add x3 add x4 add x5 ln x2", "add x0 add mul c:2 x0 ln x2", "add sin x0 add cos x1 add mul x0 x1 ln x2",
         "add x6 add x0 ln x2", "add x0 add x1 add sin x1 add cos x0 add mul x0 x1 add exp x0 add sqr x1 ln x2",
         "add mul c:1e-9 x0 add x1 ln x2", "add x0 ln x2", "add ln x2 add x0 x1"]


@pytest.mark.parametrize("n", [2000, 2049, 9001, 20011, 32768, 32769, 70001])
def test_sampled_certificate(n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-2, 2, (n, 7))
    X[: n - 5, 2] = np.abs(X[: n - 5, 2])
    X[n - 5:, 2] = -1.0  # ln x2: NaN on the last rows
    sampled = np.zeros(n, dtype=bool)
    for s in range(8):
        sampled[n * s // 8: n * s // 8 + 256] = True
    X[:, 3] = np.where(sampled, 0.0, X[:, 3])           # zero on the sample
    X[:, 4] = np.where(sampled, X[:, 0], X[:, 4])       # x0 on the sample
    X[:, 5] = np.where(sampled, X[:, 5], X[:, 0])       # x0 off the sample
    X[:, 6] = 0.0
    X[0, 6] = 1.0                                       # one row
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 3]) + 0.01 * rng.standard_normal(n)
    ods = pyoracle.OracleDataset(X, y)
    ora = ods.evaluate(encode(TREES, tuned=True), threads=4)
    for cache in (True, False):
        ctx = Context(0)
        ctx.set_mixed_min_rows(0)
        ctx.set_column_cache(cache)
        ds = ctx.dataset(X, y)
        for _ in range(2):
            dev = ds.evaluate(encode(TREES, tuned=True), PLAIN)
            for key in ("loss", "rmse", "rank"):
                assert np.array_equal(dev[key], ora[key], equal_nan=True), (key, cache)
            for a, c in zip(dev["coefs"], ora["coefs"]):
                assert np.array_equal(a, c, equal_nan=True)
        cert = ds.evaluate(encode(TREES, tuned=True), CERTIFIED)
        assert np.array_equal(cert["loss"] == 1000, ora["loss"] == 1000)
        ds.close()
        ctx.close()
