"""The sampled certificate for candidates with a NaN column, near its bound: finite
columns whose last pivots run from 1e-18 of the largest squared norm down past the
rank cut (2^-104), badly scaled and, as in Kahan's matrix, with a smallest eigenvalue
far below the last pivot, and rows outside the sample that turn the QR's order of
pivots round.  (The free term comes last, so the smallest pivot is taken after the NaN
column and never decides; a column of its size stands beside it.)  The oracle's bits:
NaN coefficients at full rank, or the rank cut."""
import numpy as np
import pytest

from oracle import pyoracle
from rils_rols_gb300.fitness import PLAIN, Context, encode

pytestmark = pytest.mark.gpu


def kahan(k, last, rng):
    """k x k upper triangle with unit first and `last` squared last diagonal entry."""
    s = last ** (0.5 / (k - 1))
    c = np.sqrt(1 - s * s)
    return (s ** np.arange(k))[:, None] * (np.eye(k) - np.triu(np.full((k, k), c * rng.uniform(0.9, 1)), 1))


@pytest.mark.parametrize("n", [9001, 20011, 40_003])
@pytest.mark.parametrize("k", [2, 5, 7])
def test_near_the_bound(n, k):
    rng = np.random.default_rng(n + k)
    sampled = np.zeros(n, dtype=bool)
    for s in range(8):
        sampled[n * s // 8: n * s // 8 + 256] = True
    y = rng.standard_normal(n)
    ranks = set()
    for e in np.linspace(-18, -34, 9):
        R = kahan(k, 10.0 ** e, rng)
        u = np.linalg.svd(R)[2][-1]
        X = rng.standard_normal((n, k)) @ R
        for turn in (False, True):
            Z = np.empty((n, k + 2))
            Z[:, :k] = X
            Z[:, k + 1] = 0.7 * 10.0 ** (e / 2) * rng.standard_normal(n)
            if turn:
                # rows along vectors across the smallest singular one, larger in the later columns
                v = np.linspace(0.1, 3, k) * rng.uniform(0.9, 1.1, k)
                v -= (v @ u) * u
                Z[~sampled, :k] = rng.standard_normal((int((~sampled).sum()), 1)) * v + 1e-3 * X[~sampled]
            Z[:, k] = 1.0
            Z[n - 3:, k] = -1.0
            trees = ["add " * (k + 1) + f"x{k + 1} " + " ".join(f"x{j}" for j in p) + f" ln x{k}"
                     for p in (range(k), range(k)[::-1], rng.permutation(k))]
            b = encode(trees, tuned=True)
            ora = pyoracle.OracleDataset(Z, y).evaluate(b, threads=3)
            ctx = Context(0)
            ds = ctx.dataset(Z, y)
            dev = ds.evaluate(b, PLAIN)
            for key in ("loss", "rmse", "size", "rank"):
                assert np.array_equal(dev[key], ora[key], equal_nan=True), (key, e, turn)
            for a, c in zip(dev["coefs"], ora["coefs"]):
                assert np.array_equal(a, c, equal_nan=True), (e, turn)
            ranks |= set(ora["rank"].tolist())
            ds.close()
            ctx.close()
    assert max(ranks) == k + 3 > min(ranks)  # both outcomes
