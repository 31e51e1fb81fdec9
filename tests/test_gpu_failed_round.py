"""A mixed round that is refused after its evaluation has started (more distinct
factor pairs than the pair cache has slots) leaves nothing behind: the next round
on the same context and dataset gives the bits of a fresh context, and the
dataset may be destroyed at once."""
import functools

import numpy as np
import pytest

from rils_rols_gb300 import _lib
from rils_rols_gb300.fitness import (_CAND_DT, _FACT_DT, CERTIFIED, MIXED, Context, EncodedBatch, encode)

pytestmark = pytest.mark.gpu
N, D, M = 8192, 3, 8           # the smallest table whose columns and pair sums are kept
FACTORS, CANDS = 12_000, 170_000
PAIR_SLOTS = 1 << 22
LDV, SIN, EMIT, MUL_CR = 1, 5, 11, 16 + 8 * 2 + 2 * 2 + 1


@functools.cache
def many_pairs():
    """CANDS sums of M of the factors sin(c_i x_j): programs LDV j, MUL c_i, SIN, EMIT."""
    rng = np.random.default_rng(5)
    f = (np.arange(M) * (FACTORS // M) + rng.integers(FACTORS // M, size=(CANDS, M))).astype(np.uint32)
    lo, hi = np.minimum(f[:, :, None], f[:, None, :]), np.maximum(f[:, :, None], f[:, None, :])
    i, j = np.triu_indices(M, 1)
    assert np.unique(lo[:, i, j].astype(np.int64) * FACTORS + hi[:, i, j]).size > PAIR_SLOTS
    code = np.empty((CANDS, M, 4), np.uint32)
    code[:, :, 0] = LDV | (f % D) << 8
    code[:, :, 1] = MUL_CR | f << 8
    code[:, :, 2] = SIN
    code[:, :, 3] = EMIT | np.arange(M, dtype=np.uint32) << 8
    cands = np.zeros(CANDS, _CAND_DT)
    cands["code_offset"] = np.arange(CANDS) * 4 * M
    cands["code_len"] = 4 * M
    cands["first_factor"] = np.arange(CANDS) * M
    cands["n_factors"] = M
    cands["mode"] = _lib.RRG_TUNED
    cands["coef_offset"] = np.arange(CANDS) * (M + 1)
    factors = np.zeros(CANDS * M, _FACT_DT)
    factors["n_nodes"] = 4
    return EncodedBatch(cands, factors, code.reshape(-1), rng.uniform(0.1, 3.0, FACTORS), CANDS * (M + 1))


def same(a, b):
    return all(np.array_equal(a[k], b[k], equal_nan=True) for k in ("loss", "rmse", "size", "rank", "flags")) and \
        all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a["coefs"], b["coefs"]))


@pytest.mark.parametrize("graph", [False, True])
def test_refused_round(graph):
    rng = np.random.default_rng(1)
    X = rng.uniform(-2, 2, (N, D))
    y = X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.01 * rng.standard_normal(N)
    trees = [f"add mul c:2 x{i % D} add sin mul c:{0.1 + i / 40!r} x{(i + 1) % D} mul x0 x{i % D}" for i in range(90)]
    good, bad = encode(trees, tuned=True), many_pairs()
    fresh = Context(0)
    dsf = fresh.dataset(X, y)
    ref = {p: dsf.evaluate(good, p) for p in (MIXED, CERTIFIED)}
    ctx = Context(0)
    ctx.set_graph(graph)
    for p in (MIXED, CERTIFIED):
        ds = ctx.dataset(X, y)
        with pytest.raises(_lib.RRGError, match="pair cache"):
            ds.evaluate(bad, p)
        assert same(ds.evaluate(good, p), ref[p])
        with pytest.raises(_lib.RRGError, match="pair cache"):
            ds.evaluate(bad, p)
        ds.close()
    for c in (dsf, fresh, ctx):
        c.close()
