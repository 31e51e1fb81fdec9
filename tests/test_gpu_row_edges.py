"""FP64 rounds at row counts around the kernels' cuts (the residual's row groups
and its four-threads-a-lane form, the QR's chunks of 16384 rows and their row
groups), one candidate at a time and many at once: the oracle's bits."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import PLAIN, Context, encode

pytestmark = pytest.mark.gpu
TREES = ["x0", "add x0 mul x1 x2", "add sin x0 add mul c:2 x1 exp x2", "add x0 add ln x1 x2", "add x0 add x0 x1",
         "add add sin x0 cos x0 add add x1 mul x1 x2 add exp mul c:0.2 x2 div x0 add c:4 x1"]


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 3, 255, 257, 2047, 2048, 2049, 8193, 16383, 16384, 16385, 18433, 32768, 49157])
def test_row_counts(ctx, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-2, 2, (n, 3))
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(n)
    ds, ods = ctx.dataset(X, y), pyoracle.OracleDataset(X, y)
    many = encode(TREES * 40 + [f"add x0 mul c:{i}.5 sin mul c:{i} x1" for i in range(60)], tuned=True)
    batches = [encode([t], tuned=True) for t in TREES] + [encode([TREES[2]], tuned=False), many]
    for b in batches:
        dev, ora = ds.evaluate(b, PLAIN), ods.evaluate(b, threads=4)
        for key in ("loss", "rmse"):
            assert np.all((dev[key] == ora[key]) | (np.isnan(dev[key]) & np.isnan(ora[key]))), (key, len(b))
        assert np.array_equal(dev["size"], ora["size"]) and np.array_equal(dev["rank"], ora["rank"])
        for a, c in zip(dev["coefs"], ora["coefs"]):
            assert np.all((a == c) | (np.isnan(a) & np.isnan(c)))
    ds.close()
