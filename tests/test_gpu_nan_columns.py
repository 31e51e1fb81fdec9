"""Factor columns with NaN rows, whose remaining rows the evaluators leave out:
the same results as the oracle (plain) and as rounds without a column cache
(mixed, certified), also when a later round reads such a factor as an operand
of min, max or a comparison, which turn NaN into numbers."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import CERTIFIED, MIXED, PLAIN, Context, encode

pytestmark = pytest.mark.gpu
# ln x0: NaN on half the rows; ln (x1 + 1.99): on one row in 400; sqrt with a NaN on row 5 or row 130 only
ROUNDS = [
    ["add ln x0 x1", "add x1 ln add x1 c:1.99", "add mul x1 x2 sqrt x3", "ln x0", "add x2 sqrt x4", "add x0 add ln x0 x0",
     "add mul x1 c:0 ln x0", "add x1 add x1 ln x0"],
    ["add max ln x0 x1 x2", "add min ln x0 x2 x1", "add lt ln x0 x1 x2", "add ln x0 x2", "max ln x0 x1", "min sqrt x3 x1",
     "add x1 max sqrt x3 x2", "add lt ln add x1 c:1.99 x0 x2", "add x0 min ln add x1 c:1.99 x2"],
    ["add ln x0 x1", "add x2 exp ln x0", "add sin ln x0 cos ln x0", "add ne ln x0 x1 eq ln x0 ln x0", "min ln x0 x1"],
]


def data(n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-2, 2, (n, 5))
    X[:, 3] = np.abs(X[:, 3])
    X[:, 4] = np.abs(X[:, 4])
    X[5, 3] = -1.0
    X[130, 4] = -1.0
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(n)
    return X, y


def bits(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return np.all((a == b) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("tuned", [True, False])
@pytest.mark.parametrize("n", [200, 3000, 9000, 40000])
def test_rounds(n, tuned):
    X, y = data(n)
    ods = pyoracle.OracleDataset(X, y)
    ctx, off = Context(0), Context(0)
    off.set_column_cache(False)
    for c in (ctx, off):
        c.set_mixed_min_rows(0)
    ds, dso = ctx.dataset(X, y), off.dataset(X, y)
    for prec in (PLAIN, CERTIFIED, MIXED):
        ctx.clear_column_cache()
        for trees in ROUNDS + ROUNDS:
            b = encode(trees, tuned=tuned)
            dev, ref = ds.evaluate(b, prec), dso.evaluate(b, prec)
            for key in ("loss", "rmse", "size", "rank", "flags"):
                assert bits(dev[key], ref[key]), (prec, key, trees)
            assert all(bits(p, q) for p, q in zip(dev["coefs"], ref["coefs"]))
            ora = ods.evaluate(b, threads=4)
            if prec == PLAIN:
                assert all(bits(dev[k], ora[k]) for k in ("loss", "rmse", "size", "rank")), trees
            assert np.array_equal(dev["loss"] == 1000, ora["loss"] == 1000), (prec, trees)
    for c in (ds, dso, ctx, off):
        c.close()
