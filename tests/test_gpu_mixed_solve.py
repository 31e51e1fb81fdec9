"""The mixed path's Gram solve, one warp a candidate, for every width it takes (1 to
8 factors): full rank, duplicate and nearly collinear factors, factors of very
different scale, and a factor with NaN rows at each position.  Certified rounds:
the oracle's sentinels, sizes and ranks, and within 1e-6 of its fitness; alone
and in a batch the same bits."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import CERTIFIED, MIXED, Context, encode

pytestmark = pytest.mark.gpu
TERMS = ["x0", "sin x1", "mul x0 x1", "exp mul c:0.3 x2", "sqr x2", "cos x0", "div x1 add c:4 x0", "mul x1 x2"]


def tree(terms):
    return "add " * (len(terms) - 1) + " ".join(terms)


def batch(m):
    t = TERMS[:m]
    out = [tree(t), tree([f"mul c:1e-6 {t[0]}"] + t[1:]), tree(t[:-1] + ["mul x0 add c:1 mul c:1e-9 x1"]),
           tree(t[:-1] + ["mul c:1e5 sqr x0"])]
    out += [tree(t[:i] + ["ln x3"] + t[i + 1:]) for i in range(m)]
    if m > 1:
        out += [tree(t[:-1] + [t[0]]), tree(t[:-1] + ["sin c:1"])]
    return out


@pytest.mark.parametrize("m", range(1, 9))
def test_widths(m):
    n = 5003
    rng = np.random.default_rng(m)
    X = rng.uniform(-2, 2, (n, 4))
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.3 * X[:, 0] + 0.01 * rng.standard_normal(n)
    ctx = Context(0)
    ctx.set_mixed_min_rows(0)
    ctx.set_column_cache(False)
    ds, ods = ctx.dataset(X, y), pyoracle.OracleDataset(X, y)
    trees = batch(m)
    for prec in (MIXED, CERTIFIED):
        dev = ds.evaluate(encode(trees, tuned=True), prec)
        for i, t in enumerate(trees):
            one = ds.evaluate(encode([t], tuned=True), prec)
            assert all(np.array_equal(one[k], dev[k][i:i + 1], equal_nan=True) for k in ("loss", "rmse", "rank")), t
    ora = ods.evaluate(encode(trees, tuned=True), threads=4)
    sent = ora["loss"] == 1000
    assert np.array_equal(dev["loss"] == 1000, sent)
    for key in ("size", "rank"):
        assert np.array_equal(dev[key][~sent], ora[key][~sent]), key
    fv = lambda r: (1 + r["loss"]) * (1 + r["rmse"]) * (1 + 1e-3 * r["size"])  # noqa: E731
    ok = ~sent & np.isfinite(fv(ora))
    assert (np.abs(fv(dev)[ok] - fv(ora)[ok]) / fv(ora)[ok]).max() <= 1e-6
    ds.close()
    ctx.close()
