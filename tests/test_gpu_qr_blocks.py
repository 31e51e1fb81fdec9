"""The one-block column-pivoted QR at every block width (a lone candidate, some,
and many), with the working columns in shared memory and, where they do not fit,
in the scratch, at row counts around its 32-lane groups and 256-row strides, with
narrow and wide candidates, rank cuts and NaN columns: the oracle's bits."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import PLAIN, Context, encode

pytestmark = pytest.mark.gpu
_T9 = ["x0", "x1", "x2", "sin x0", "cos x1", "mul x0 x1", "exp mul c:0.3 x2", "div x0 add c:4 x1", "sqr x2"]
_T20 = _T9 + ["sin x1", "sin x2", "cos x0", "cos x2", "mul x1 x2", "mul x0 x2", "sqr x0", "sqr x1", "sin mul x0 x1",
              "cos mul x1 x2", "exp mul c:0.2 x0"]
_T35 = _T20 + [f"sin mul c:{i}.5 x{i % 3}" for i in range(2, 17)]
NARROW = ["x0", "add x0 mul x1 x2", "add sin x0 add x0 sin x0", "add x0 add mul x0 add c:1 mul c:1e-9 x1 x2",
          "add x0 add ln x1 x2", "add x0 mul c:0 x1", "add exp mul c:800 x0 x1"]
WIDE = ["add " * (len(t) - 1) + " ".join(t) for t in (_T9, _T20, _T35)]


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def check(ods, ds, trees):
    b = encode(trees, tuned=True)
    dev, ora = ds.evaluate(b, PLAIN), ods.evaluate(b, threads=8)
    for key in ("loss", "rmse"):
        assert np.all((dev[key] == ora[key]) | (np.isnan(dev[key]) & np.isnan(ora[key]))), key
    assert np.array_equal(dev["size"], ora["size"]) and np.array_equal(dev["rank"], ora["rank"])
    for t, a, c in zip(trees, dev["coefs"], ora["coefs"]):
        assert np.all((a == c) | (np.isnan(a) & np.isnan(c))), t


# with 3 to 37 columns: shared memory up to about 9000 to 700 rows
@pytest.mark.parametrize("n", [2, 31, 33, 150, 257, 569, 700, 1025, 6001, 16384])
def test_block_widths(ctx, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-2, 2, (n, 3))
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(n)
    ds, ods = ctx.dataset(X, y), pyoracle.OracleDataset(X, y)
    for t in NARROW + WIDE:
        check(ods, ds, [t])
    some = [f"add x0 mul c:{i}.5 sin mul c:{i} x1" for i in range(1, 400)]
    check(ods, ds, some + NARROW + WIDE)
    if n <= 1025:
        check(ods, ds, [f"add sin mul c:{i} x0 add cos mul c:{i}.5 x1 mul x{i % 3} exp mul c:{i}e-4 x2"
                        for i in range(2500)] + NARROW)
    ds.close()
