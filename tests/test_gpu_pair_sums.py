"""The factor table's cross sums, four partners folded together, at row counts
around a block of 4096 rows and at 1 to 18 partners of one factor (some with NaN
rows): within the certified form's 1e-6 of the oracle, and the same bits when the
batch is reversed (the other factor of a pair held, other partners beside it)."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import CERTIFIED, MIXED, Context, encode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("partners", [1, 2, 3, 4, 5, 16, 17, 18])
@pytest.mark.parametrize("n", [300, 4095, 4097, 8192, 12289])
def test_partners(n, partners):
    rng = np.random.default_rng(n + partners)
    X = rng.uniform(-2, 2, (n, 3))
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(n)
    trees = [f"add x0 sin mul c:{i + 1}.25 x1" for i in range(partners)]
    trees += ["add x0 ln x1", "add ln x1 mul x0 x2", "add add x2 exp x1 add cos x0 mul x1 x2", "mul x0 x1"]
    ctx = Context(0)
    ctx.set_mixed_min_rows(0)
    ds, ods = ctx.dataset(X, y), pyoracle.OracleDataset(X, y)
    ora = ods.evaluate(encode(trees, tuned=True), threads=4)
    for prec in (MIXED, CERTIFIED):
        ctx.clear_column_cache()
        fwd = ds.evaluate(encode(trees, tuned=True), prec)
        ctx.clear_column_cache()
        rev = ds.evaluate(encode(trees[::-1], tuned=True), prec)
        for key in ("loss", "rmse"):
            a, b = np.asarray(fwd[key]), np.asarray(rev[key])[::-1]
            assert np.all((a == b) | (np.isnan(a) & np.isnan(b))), (prec, key)
        sent = ora["loss"] == 1000
        assert np.array_equal(fwd["loss"] == 1000, sent)
        if prec == CERTIFIED:
            fv = lambda r: (1 + r["loss"]) * (1 + r["rmse"]) * (1 + 1e-3 * r["size"])  # noqa: E731
            ok = ~sent & np.isfinite(fv(ora))
            assert (np.abs(fv(fwd)[ok] - fv(ora)[ok]) / fv(ora)[ok]).max() <= 1e-6
    ds.close()
    ctx.close()
