"""FP64 columns that a re-scoring kept in part (no program read them as an operand, so
rows after a NaN may be missing) and a later round reads as operands: that round
evaluates them, the whole columns take the kept ones' place, and the rounds after it
evaluate nothing again.  Results are those of a context that keeps no columns."""
import numpy as np
import pytest

from rils_rols_gb300.fitness import CERTIFIED, Context, encode

pytestmark = pytest.mark.gpu
N, D, K = 40_000, 3, 80


def same(a, b):
    return all(np.array_equal(a[k], b[k], equal_nan=True) for k in ("loss", "rmse", "size", "rank", "flags")) and \
        all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a["coefs"], b["coefs"]))


@pytest.mark.parametrize("nan", [False, True])
def test_whole_columns_take_their_place(nan):
    rng = np.random.default_rng(9)
    X = rng.uniform(0.5, 2, (N, D))
    if nan:
        X[300:, 2] -= 40.0
    y = X[:, 0] * X[:, 1] + 0.1 * rng.standard_normal(N)
    # every candidate holds the same factor twice: a rank cut, which the FP64 path scores
    dup = [f"add mul c:2 sin add c:{i / 16!r} x0 mul c:3 sin add c:{i / 16!r} x0" for i in range(K)]
    t = [f"ln add c:{3 + i / 16!r} x2" for i in range(K)]
    alone = [f"add {a} {b}" for a, b in zip(dup, t)]
    first = encode(alone, tuned=True)
    top = encode(alone + [f"add {a} max {b} x1" for a, b in zip(dup, t)], tuned=True)
    low = encode(alone + [f"add {a} min {b} x1" for a, b in zip(dup, t)], tuned=True)
    ctx, plain = Context(0), Context(0)
    plain.set_column_cache(False)
    ds, dsp = ctx.dataset(X, y), plain.dataset(X, y)

    def columns(b):
        """FP64 columns the round's re-scoring evaluated."""
        assert same(ds.evaluate(b, CERTIFIED), dsp.evaluate(b, CERTIFIED))
        assert ctx.last_round_stats()["fp64_rescored"] == len(b)
        return round(ctx.last_round_bytes()["fp64_eval"] / (8 * N)) - D

    assert columns(first) == 2 * K
    assert columns(first) == 0
    assert columns(top) == 2 * K      # the logarithms, read by max as well, and max
    assert columns(top) == 0
    assert columns(low) == K          # min alone
    assert columns(first) == 0 and columns(top) == 0
    for c in (ds, dsp, ctx, plain):
        c.close()
