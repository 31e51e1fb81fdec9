"""No trial of shapes that are the same launch: nothing is timed or stored, and the
round takes its usual form.  Wide levels of FP64 columns run in pieces that the rows
decide, whatever the tuner's waves; groups of factors are timed in the sizes that a round
large enough for them would use."""
import numpy as np
import pytest

from rils_rols_gb300.fitness import CERTIFIED, MIXED, PLAIN, Context, encode, tune_mode, tune_report, tune_reset

pytestmark = pytest.mark.gpu
N, D = 100_000, 4


@pytest.fixture()
def ds():
    rng = np.random.default_rng(4)
    X = rng.uniform(-1, 1, (N, D))
    ctx = Context(0)
    ctx.set_column_cache(False)
    d = ctx.dataset(X, X[:, 0] * X[:, 1] + 0.1 * rng.standard_normal(N))
    yield d
    tune_reset()
    tune_mode(True)
    d.close()
    ctx.close()


def factors(k):
    return [f"mul x{i % D} add c:{i / 64!r} x{(i + 1) % D}" for i in range(k)]


def knobs(ds, b, prec):
    tune_reset()
    tune_mode(True)
    out = ds.evaluate(b, prec)
    return out, ds.ctx.last_round_launches(), {e["knob"] for e in tune_report()}


def test_wide_level_of_fp64_columns(ds):
    b = encode(factors(400), tuned=True)  # 25 pieces of rows a column; 16 waves are 7 blocks a column
    tune_mode(False)
    ref = ds.evaluate(b, PLAIN)
    launches = ds.ctx.last_round_launches()
    out, ran, rep = knobs(ds, b, PLAIN)
    assert rep == set() and ran == launches
    assert np.array_equal(out["loss"], ref["loss"]) and np.array_equal(out["rmse"], ref["rmse"])
    # a narrow level of the same rows is timed
    assert knobs(ds, encode(factors(12), tuned=True), PLAIN)[2] == {"eval_waves"}


@pytest.mark.parametrize("prec", [MIXED, CERTIFIED])
def test_factor_groups(ds, prec):
    b = encode(factors(14), tuned=True)  # at most 16 factors: one group in every size
    tune_mode(False)
    ref = ds.evaluate(b, prec)
    out, _, rep = knobs(ds, b, prec)
    assert "fac_group" not in rep
    assert np.array_equal(out["loss"], ref["loss"]) and np.array_equal(out["rmse"], ref["rmse"])
    # the sizes differ from 17 factors on, though 48 are few for 16 to a block
    b = encode(factors(48), tuned=True)
    tune_mode(False)
    ref = ds.evaluate(b, prec)
    out, _, rep = knobs(ds, b, prec)
    assert "fac_group" in rep
    e = next(e for e in tune_report() if e["knob"] == "fac_group")
    # 48 factors in one block take longer than in three; as one and the same launch they would not
    assert set(e["ms"]) == {64, 32, 16} and e["ms"][64] > 1.3 * e["ms"][16], e
    assert np.array_equal(out["loss"], ref["loss"]) and np.array_equal(out["rmse"], ref["rmse"])
