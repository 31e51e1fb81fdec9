"""The tuner's trials on columns that hold a NaN: every shape evaluates the same rows.
All columns here are NaN in the last row alone.  A shape that found the mark of the
shape before it would leave nearly every row out and be timed many times shorter;
the shapes themselves differ by less than half."""
import numpy as np
import pytest

from rils_rols_gb300.fitness import (CERTIFIED, MIXED, PLAIN, Context, encode, tune_mode, tune_report, tune_reset)

pytestmark = pytest.mark.gpu
N, D = 400_000, 4


@pytest.fixture(scope="module")
def problem():
    rng = np.random.default_rng(2)
    X = rng.uniform(0.5, 2, (N, D))
    X[-1] = -30.0
    y = X[:, 0] * X[:, 1] + 0.1 * rng.standard_normal(N)
    # 12 columns of one level: few enough that the waves decide the blocks
    chain = "exp sin exp cos exp sin " * 2
    return X, y, [f"mul {chain}add c:{i / 9!r} x{i % D} ln add c:{i / 8!r} x{(i + 1) % D}" for i in range(12)]


@pytest.mark.parametrize("prec", [PLAIN, MIXED, CERTIFIED])
def test_every_shape_evaluates_the_same_rows(problem, prec):
    X, y, trees = problem
    b = encode(trees, tuned=False)
    ctx = Context(0)
    ctx.set_column_cache(False)
    ds = ctx.dataset(X, y)
    try:
        tune_mode(False)
        ref = ds.evaluate(b, prec)
        tune_reset()
        tune_mode(True)
        out = ds.evaluate(b, prec)
        for k in ("loss", "rmse", "size", "rank", "flags"):
            assert np.array_equal(out[k], ref[k], equal_nan=True), k
        for e in tune_report():
            assert max(e["ms"].values()) < 2.5 * min(e["ms"].values()), e
        if prec == PLAIN:
            assert [e["knob"] for e in tune_report()] == ["eval_waves"]
    finally:
        tune_reset()
        tune_mode(True)
        ds.close()
        ctx.close()
