"""The probe of the mixed path (both interpreters on up to 1024 rows, one block
per factor) around its row and thread counts, with factors that are NaN, infinite
or beyond FP32 on some rows: the oracle's sentinels and sizes, and within the
certified form's 1e-6 of it."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import CERTIFIED, Context, encode

pytestmark = pytest.mark.gpu
TREES = ["add x0 mul x1 x2", "add ln x0 x1", "add x1 sqrt x3", "add exp mul c:60 x0 x1", "add x2 exp mul c:400 x1",
         "add x0 div x1 sub x2 x2", "add sin x0 mul c:2 cos x1", "mul x0 x1", "sub mul x0 x1 sin x2"]


@pytest.mark.parametrize("tuned", [True, False])
@pytest.mark.parametrize("n", [2, 31, 511, 513, 1023, 1024, 1025, 2049])
def test_probe_rows(n, tuned):
    rng = np.random.default_rng(n)
    X = rng.uniform(-2, 2, (n, 4))
    X[:, 3] = np.abs(X[:, 3])
    X[-1, 3] = -1.0  # sqrt x3: NaN on the last row only
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(n)
    ctx = Context(0)
    ctx.set_mixed_min_rows(0)
    ds, ods = ctx.dataset(X, y), pyoracle.OracleDataset(X, y)
    b = encode(TREES, tuned=tuned)
    cert, ora = ds.evaluate(b, CERTIFIED), ods.evaluate(b, threads=4)
    sent = ora["loss"] == 1000
    assert np.array_equal(cert["loss"] == 1000, sent)
    assert np.array_equal(cert["size"][~sent], ora["size"][~sent])
    fv = lambda r: (1 + r["loss"]) * (1 + r["rmse"]) * (1 + 1e-3 * r["size"])  # noqa: E731
    ok = ~sent & np.isfinite(fv(ora))
    assert (np.abs(fv(cert)[ok] - fv(ora)[ok]) / fv(ora)[ok]).max(initial=0.0) <= 1e-6
    ds.close()
    ctx.close()
