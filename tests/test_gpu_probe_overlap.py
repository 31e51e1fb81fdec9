"""The factor probe runs beside the evaluation in every mixed round without a
launch-shape trial, also while a shape is still open because no round has carried
enough work to time it: such a round takes the device time of the same round with
the tuner off."""
import numpy as np
import pytest

from rils_rols_gb300.fitness import CERTIFIED, Context, encode, tune_mode, tune_report, tune_reset

pytestmark = pytest.mark.gpu
N, D = 50_000, 30


def test_open_shape_costs_nothing():
    rng = np.random.default_rng(7)
    X = rng.uniform(-1, 1, (N, D))
    y = X[:, 0] * X[:, 1] + 0.1 * rng.standard_normal(N)
    # one candidate of eight long factors (0.4M row-columns; a shape is timed from 1M on)
    chain = "sin exp cos exp " * 4
    b = encode(["add " * 7 + " ".join(f"mul x{3 * i} {chain}mul c:{0.2 + i / 16!r} x{3 * i + 1}" for i in range(8))])
    ctx = Context(0)
    ctx.set_timing(True)
    ds = ctx.dataset(X, y)

    def block():
        t = []
        for _ in range(60):
            ctx.clear_column_cache()
            ds.evaluate(b, CERTIFIED)
            t.append(sum(v[0] for v in ctx.last_round_timing().values()))
        return float(np.median(t))

    try:
        t = {True: [], False: []}
        for _ in range(4):
            for on in t:
                tune_reset()
                tune_mode(on)
                t[on].append(block())
                assert all(e["knob"] != "fac_stage" for e in tune_report())  # still open
        # the probe in series adds a fifth or more; medians of one form differ by a few percent
        assert min(t[True]) < 1.1 * min(t[False]), t
    finally:
        tune_reset()
        tune_mode(True)
        ds.close()
        ctx.close()
