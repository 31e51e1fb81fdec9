"""Batches of many unlike trees over one dataset, whose shared columns are left
out once no factor needs them: the same results as the same trees in batches too
small for that, and a sample of them against the oracle's bits.  NaN rows lie in
the first rows, just beyond them and late; min, max and comparisons read columns
with NaN as operands."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300 import synth
from rils_rols_gb300.fitness import CERTIFIED, MIXED, PLAIN, Context, encode

pytestmark = pytest.mark.gpu
N, TREES = 70_001, 1600  # about 1500 shared columns


@pytest.fixture(scope="module")
def problem():
    rng = np.random.default_rng(11)
    X = rng.uniform(0.1, 2, (N, 5))
    X[N // 2:, 2] -= 1.0            # ln x2, sqrt x2: NaN from the middle on
    for j, r in ((3, 1023), (4, 1024)):
        X[r, j] = -1.0              # NaN on one row, the last of the first rows and the one after
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(N)
    binary = synth.BINARY + synth.CLS_BINARY
    trees = [synth.random_tree(rng, int(rng.integers(5, 40)), 5, binary=binary if i % 2 else synth.BINARY)
             for i in range(TREES)]
    return X, y, trees


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return np.all((a == b) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("cache", [True, False])
@pytest.mark.parametrize("prec", [PLAIN, MIXED, CERTIFIED])
def test_many_trees(problem, prec, cache):
    X, y, trees = problem
    ctx, small = Context(0), Context(0)
    small.set_column_cache(False)
    ctx.set_column_cache(cache)
    ds, dsm = ctx.dataset(X, y), small.dataset(X, y)
    ds.evaluate(encode(trees[:64], tuned=True), prec)
    for _ in range(2):  # the second time with what the first one kept
        dev = ds.evaluate(encode(trees, tuned=True), prec)
    step = 160
    for i in range(0, TREES, step):
        ref = dsm.evaluate(encode(trees[i:i + step], tuned=True), prec)
        for key in ("loss", "rmse", "size", "rank"):
            assert same(dev[key][i:i + step], ref[key]), (key, i)
        assert all(same(a, b) for a, b in zip(dev["coefs"][i:i + step], ref["coefs"]))
    if prec == PLAIN and cache:
        ora = pyoracle.OracleDataset(X, y).evaluate(encode(trees[::16], tuned=True), threads=8)
        assert all(same(dev[k][::16], ora[k]) for k in ("loss", "rmse", "size", "rank"))
    for c in (ds, dsm, ctx, small):
        c.close()
