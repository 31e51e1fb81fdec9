"""Every operator of the FP64 evaluator on the device, on random significands,
operands next to half-way points and special values: the oracle's bits."""
import numpy as np
import pytest

from test_fp64_int_cpu import operands

pytestmark = pytest.mark.gpu
TREES = {"mul": "mul x0 x1", "div": "div x0 x1", "sqrt": "sqrt x0", "sqr": "sqr x0", "lt": "lt x0 x1",
         "eq": "eq x0 x1", "ne": "ne x0 x1", "min": "min x0 x1", "max": "max x0 x1", "sin": "sin x0",
         "cos": "cos x0", "log": "ln x0", "exp": "exp x0"}


@pytest.mark.parametrize("op", sorted(TREES))
def test_operator_bits(op):
    from oracle import pyoracle
    from rils_rols_gb300.fitness import Context, encode
    a, b = operands(op, 7, 40_000)
    if op in ("sin", "cos", "log", "exp"):
        a = np.concatenate([a, np.random.default_rng(7).uniform(-40, 40, 20_000), np.arange(-500, 500) * (np.pi / 4)])
        b = np.resize(b, len(a))
    X, y = np.stack([a, b], axis=1), np.arange(len(a), dtype=np.float64)
    ref = pyoracle.OracleDataset(X, y).predict(encode([TREES[op]], tuned=False))
    ctx = Context(0)
    ds = ctx.dataset(X, y)
    got = ds.predict(TREES[op])
    ds.close()
    ctx.close()
    same = (got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), (op, X[~same][:3], got[~same][:3], ref[~same][:3])
