"""The two-part evaluation of a table with many shared columns (the first 1024 rows
of every level, then the other rows of what still counts): the number of launches
shows that it ran, in the FP64 table, the double-float table and the re-scoring
lane; results are those of the same trees in batches too small for it, and a sample
has the oracle's bits.  Features turn negative (NaN under ln and sqrt) on single rows
at the edges of the first rows and of the rows that are always evaluated, and from
the middle on; comparisons, minima and maxima read columns with NaN as operands."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300 import synth
from rils_rols_gb300.fitness import CERTIFIED, MIXED, PLAIN, Context, encode, tune_mode

pytestmark = pytest.mark.gpu
# the second part needs shared columns x rows >= 2^26 and every fourth column shared
N, N_BELOW, D, TREES, STEP = 120_001, 40_001, 7, 2000, 200


@pytest.fixture(scope="module")
def problem():
    rng = np.random.default_rng(11)
    X = rng.uniform(0.1, 2, (N, D))
    X[N // 2:, 2] -= 1.0
    for j, r in ((3, 1023), (4, 1024), (5, 127), (6, 128)):
        X[r, j] = -1.0
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(N)
    binary = synth.BINARY + synth.CLS_BINARY
    trees = [synth.random_tree(rng, int(rng.integers(5, 50)), D, binary=binary if i % 2 else synth.BINARY, p_var=0.8)
             for i in range(TREES)]
    tune_mode(False)
    yield X, y, trees
    tune_mode(True)


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return np.all((a == b) | (np.isnan(a) & np.isnan(b)))


def launches(X, y, trees, prec, n):
    ctx = Context(0)
    ctx.set_column_cache(False)
    ds = ctx.dataset(X[:n], y[:n])
    ds.evaluate(encode(trees, tuned=True), prec)
    k = ctx.last_round_launches()
    ds.close()
    ctx.close()
    return k


def test_runs_in_two_parts(problem):
    X, y, trees = problem
    more = {p: launches(X, y, trees, p, N) - launches(X, y, trees, p, N_BELOW) for p in (PLAIN, MIXED, CERTIFIED)}
    # a second launch for every level and one between: in a plain round for one table, in a mixed one for two
    assert more[PLAIN] >= 3 and more[MIXED] >= 2 * more[PLAIN] and more[CERTIFIED] >= 2 * more[PLAIN], more
    assert launches(X, y, trees[:STEP], PLAIN, N) - launches(X, y, trees[:STEP], PLAIN, N_BELOW) == 0


@pytest.mark.parametrize("cache", [False, True])
@pytest.mark.parametrize("prec", [PLAIN, MIXED, CERTIFIED])
def test_same_results(problem, prec, cache):
    X, y, trees = problem
    ctx, small = Context(0), Context(0)
    ctx.set_column_cache(cache)
    small.set_column_cache(False)
    ds, dsm = ctx.dataset(X, y), small.dataset(X, y)
    batch = encode(trees, tuned=True)
    rounds = [ds.evaluate(batch, prec) for _ in range(2)]  # the second with what the first one kept
    for i in range(0, TREES, STEP):
        ref = dsm.evaluate(encode(trees[i:i + STEP], tuned=True), prec)
        for dev in rounds:
            for key in ("loss", "rmse", "size", "rank"):
                assert same(dev[key][i:i + STEP], ref[key]), (key, i)
            assert all(same(a, b) for a, b in zip(dev["coefs"][i:i + STEP], ref["coefs"]))
    if prec == PLAIN:
        ora = pyoracle.OracleDataset(X, y).evaluate(encode(trees[::20], tuned=True), threads=8)
        assert all(same(rounds[0][k][::20], ora[k]) for k in ("loss", "rmse", "size", "rank"))
    for c in (ds, dsm, ctx, small):
        c.close()
