"""Factors that share deep nestings of transcendental functions: a round takes
time in proportion to the depth (finding equal subtrees compares every node once),
and gives the results of the same candidates scored one at a time."""
import time

import numpy as np
import pytest

from rils_rols_gb300.fitness import PLAIN, Context, encode

pytestmark = pytest.mark.gpu
N, D, K = 300, 6, 40


def batch(depth):
    chain = " ".join(["sin"] * depth)
    return [f"mul x{i % D} add c:{i / 8!r} {chain} x{i // D % D}" for i in range(K)]


@pytest.fixture(scope="module")
def ds():
    rng = np.random.default_rng(3)
    X = rng.uniform(-2, 2, (N, D))
    ctx = Context(0)
    d = ctx.dataset(X, X[:, 0] * X[:, 1] - np.sin(X[:, 2]) + 0.1 * rng.standard_normal(N))
    yield d
    d.close()
    ctx.close()


def test_time_follows_depth(ds):
    t = {}
    for depth in (250, 1000):
        b = encode(batch(depth), tuned=True)
        ds.evaluate(b, PLAIN)
        runs = []
        for _ in range(9):
            t0 = time.perf_counter()
            ds.evaluate(b, PLAIN)
            runs.append(time.perf_counter() - t0)
        t[depth] = min(runs)
    # four times the nodes and launches; 16 times the comparisons if each chain is walked to its end
    assert t[1000] < 8 * t[250], t


@pytest.mark.parametrize("depth", [1, 2, 33, 120])
def test_same_as_alone(ds, depth):
    trees = batch(depth)
    both = ds.evaluate(encode(trees, tuned=True), PLAIN)
    for i in range(0, K, 7):
        one = ds.evaluate(encode(trees[i:i + 1], tuned=True), PLAIN)
        for k in ("loss", "rmse", "size", "rank"):
            assert one[k][0] == both[k][i], (k, i)
        assert np.array_equal(one["coefs"][0], both["coefs"][i])
