"""The workloads whose speed this repository answers for, as measurable cases.

A case is a dict of plain values; prepare() builds what a caller holds before
the call (host data made from the seed, the dataset resident on the device,
the encoded candidate batches), run() makes one pass through the public entry
points, exact() restates a round in 64-bit numpy from the batch alone, and
work() counts what a pass cannot do without.  Three kinds:

  round    rounds of candidates on one resident dataset, submitted and waited
           for one after another (rrg_round_submit / rrg_round_wait), as the
           search submits them.  The column cache is emptied at the start of a
           pass: a pass stands for rounds on data the context has not seen.
  single   one tuned candidate, the form of a local search's first scoring and
           of the re-scoring after every accepted move;
  fit      a whole fit through the drop-in class, then predict on the same
           rows.

Problems: "model" (a sum of products, sines, exponentials and quotients of the
features plus noise; the candidates are the local-search neighbourhood of
models on the way to it), "class" (correlated lognormal features, 0/1 labels,
the classifier's operators) and "trees" (random expression trees of 3 to 50
nodes, the batched-fitness workload).
"""
from __future__ import annotations

import functools
import math
import random
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "rils-rols_gb300"))

from rils_rols_gb300 import synth  # noqa: E402
from rils_rols_gb300.fitness import (CERTIFIED, MIXED, PLAIN, Context, candidates, encode,  # noqa: E402
                                     result_dtype)

PRECISION = {"plain": PLAIN, "mixed": MIXED, "certified": CERTIFIED}


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest call: one candidate on a table of 150 rows (the toy problem's training split)
        {"name": "single_150_plain", "kind": "single", "problem": "model", "n": 150, "d": 2, "stage": 3,
         "precision": "plain"},
        # the start and the re-score of every local search on a large table, in the drop-in's default arithmetic
        {"name": "single_1m_plain", "kind": "single", "problem": "model", "n": 1_000_000, "d": 5, "stage": 4,
         "precision": "plain"},
        # a classifier's local-search round on a clinical-sized table (569 x 30)
        {"name": "class_569_plain", "kind": "round", "problem": "class", "n": 569, "d": 30, "stages": "2",
         "tuned": True, "precision": "plain"},
        # the same estimator's whole fit and prediction, where launches, waits and host work count
        {"name": "class_fit_569", "kind": "fit", "problem": "class", "n": 569, "d": 30, "calls": 10_000,
         "precision": "plain"},
        # a mid-sized table of odd length, three features, default arithmetic
        {"name": "round_20011_plain", "kind": "round", "problem": "model", "n": 20_011, "d": 3, "stages": "4",
         "tuned": True, "precision": "plain"},
        # many features, odd length, the throughput form without certificate
        {"name": "round_50021_mixed", "kind": "round", "problem": "model", "n": 50_021, "d": 20, "stages": "2",
         "tuned": True, "precision": "mixed"},
        # the untuned perturbations that open every iteration of a search
        {"name": "perturb_99991_certified", "kind": "round", "problem": "model", "n": 99_991, "d": 9, "stages": "4",
         "tuned": False, "precision": "certified"},
        # batched fitness of random trees, default arithmetic
        {"name": "trees_100k_plain", "kind": "round", "problem": "trees", "n": 100_000, "d": 10, "trees": 2048,
         "tuned": True, "precision": "plain"},
        # batched fitness of random trees, the full 8192, certified
        {"name": "trees_100k_certified", "kind": "round", "problem": "trees", "n": 100_000, "d": 10, "trees": 8192,
         "tuned": True, "precision": "certified"},
        # one local-search round at a million rows in the default arithmetic
        {"name": "round_1m_plain", "kind": "round", "problem": "model", "n": 1_000_000, "d": 5, "stages": "2",
         "tuned": True, "precision": "plain"},
        # the headline: eight rounds of a search at a million rows, certified, columns kept between them
        {"name": "search_1m_certified", "kind": "round", "problem": "model", "n": 1_000_000, "d": 5,
         "stages": "01234567", "tuned": True, "precision": "certified"},
        # a whole certified regression fit and prediction on 200k rows
        {"name": "fit_200k_certified", "kind": "fit", "problem": "model", "n": 200_000, "d": 5, "calls": 20_000,
         "precision": "certified"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "round", "round", "round", "trees", "trees", "fit"])
    prec = rng.choice(["plain", "plain", "mixed", "certified", "certified"])
    if kind == "single":
        return {"kind": "single", "problem": "model", "n": _log_uniform(rng, 150, 1_000_000), "d": rng.randint(2, 20),
                "stage": rng.randint(0, 7), "precision": prec}
    if kind == "fit":
        problem = rng.choice(["model", "class"])
        return {"kind": "fit", "problem": problem, "n": _log_uniform(rng, 150, 100_000), "d": rng.randint(3, 12),
                "calls": _log_uniform(rng, 1_000, 10_000), "precision": prec}
    if kind == "trees":
        n = _log_uniform(rng, 500, 300_000)
        return {"kind": "round", "problem": "trees", "n": n, "d": rng.randint(2, 20),
                "trees": _log_uniform(rng, 64, min(4096, max(128, 400_000_000 // n))), "tuned": rng.random() < 0.8,
                "precision": prec}
    if rng.random() < 0.25:
        return {"kind": "round", "problem": "class", "n": _log_uniform(rng, 300, 30_000), "d": rng.randint(4, 30),
                "stages": rng.choice("012"), "tuned": rng.random() < 0.7, "precision": prec}
    n = _log_uniform(rng, 1_000, 1_000_000)
    top = 2 if n > 300_000 else 4 if n > 100_000 else 7  # the neighbourhood grows with the model and with d
    stages = "".join(str(rng.randint(0, top)) for _ in range(1 if prec == "plain" else rng.randint(1, 3)))
    return {"kind": "round", "problem": "model", "n": n, "d": rng.randint(2, 6 if n > 300_000 else 16),
            "stages": stages, "tuned": rng.random() < 0.75, "precision": prec}


# ----------------------------------------------------------------- inputs --
def _term(rng, d):
    """One additive term of a generating model, in prefix form."""
    a, b = rng.randrange(d), rng.randrange(d)
    c = rng.choice([-1, 1]) * rng.uniform(0.5, 3.0)
    return rng.choice([
        f"mul c:{c!r} mul x{a} x{b}", f"mul c:{c!r} sin x{a}", f"mul c:{c!r} exp mul c:{rng.uniform(0.2, 0.4)!r} x{a}",
        f"mul c:{c!r} div sin x{a} add c:1 mul x{b} x{b}", f"mul c:{c!r} x{a}"])


def _stages(rng, d):
    """Eight models on the way to a generating formula of three terms, the last
    one the formula: a product, then with an offset, then with an exponential
    (its constant still off in one of them), a sine and a quotient, as a search
    passes them."""
    v = [i % d for i in range(5)]
    k = [rng.uniform(0.8, 1.2) for _ in range(4)]
    p = f"mul c:{2.5 * k[0]!r} mul x{v[0]} x{v[1]}"
    e = f"mul c:{0.7 * k[1]!r} exp mul c:{0.3 * k[2]!r} x{v[4]}"
    q = f"div sin x{v[2]} add c:1 sqr x{v[3]}"
    truth = f"sub add {p} {e} div sin x{v[2]} add c:1 mul x{v[3]} x{v[3]}"
    return truth, [p, f"add {p} c:{k[3]!r}", f"add {p} {e}", f"add {p} mul c:0.93 exp x{v[4]}",
                   f"add add {p} {e} mul c:-0.98 sin x{v[2]}", f"add add {p} {e} mul c:-1 {q}",
                   f"add add {p} {e} div sin x{v[2]} sqr x{v[3]}", truth]


def _class_stages(rng, d):
    v = [i % d for i in range(4)]
    c = [rng.uniform(0.3, 2.0) for _ in range(3)]
    truth = f"sub add mul c:{c[0]!r} x{v[0]} lt x{v[1]} c:{c[1]!r} add x{v[2]} mul c:0.1 x{v[3]}"
    return truth, [f"mul c:{c[0]!r} x{v[0]}", f"add mul c:{c[0]!r} x{v[0]} lt x{v[1]} c:{c[1]!r}",
                   f"add mul c:{c[0]!r} x{v[0]} add lt x{v[1]} c:{c[1]!r} mul c:{c[2]!r} x{v[2]}"]


def _random_tree(rng, size, d):
    """A random expression of exactly `size` nodes (the operators, leaves and
    constants of synth.random_tree)."""
    out, todo = [], [size]
    while todo:
        s = todo.pop()
        if s == 1:
            out.append(f"x{rng.randrange(d)}" if rng.random() < 0.5 else f"c:{rng.uniform(-5.0, 5.0)!r}")
            continue
        op = rng.choice(synth.UNARY + synth.BINARY if s >= 3 else synth.UNARY)
        out.append(op)
        if op in synth.UNARY:
            todo.append(s - 1)
        else:
            left = rng.randint(1, s - 2)
            todo += [s - 1 - left, left]
    return " ".join(out)


def _problem(case, seed):
    """Host data (X, y) and the rounds of prefix trees of a case."""
    rng, gen = random.Random(seed), np.random.default_rng(seed)
    n, d = case["n"], case["d"]
    if case["problem"] == "class":
        X = np.exp(math.sqrt(0.5) * (gen.standard_normal((n, d)) + gen.standard_normal((n, 1))))
        truth, stages = _class_stages(rng, d)
        v = synth.eval_tree(truth, X)
        y = (v > np.median(v)).astype(np.float64)
        flip = gen.random(n) < 0.05
        y[flip] = 1.0 - y[flip]
    else:
        if case["problem"] == "trees":
            X = gen.standard_normal((n, d))
            truth, stages = " ".join(["add"] * 2 + [_term(rng, d) for _ in range(3)]), []
        else:
            # untuned values are compared as they are: a range in which no
            # perturbation's square leaves FP64's
            r = 3.0 if case.get("tuned", True) else 1.0
            X = gen.uniform(-r, r, (n, d))
            truth, stages = _stages(rng, d)
        y = synth.eval_tree(truth, X)
        y = y + gen.normal(0.0, 0.005 * np.std(y), n)
    if case["kind"] == "fit":
        return X, y, []
    if case["problem"] == "trees":
        return X, y, [[_random_tree(rng, rng.randint(3, 50), d) for _ in range(case["trees"])]]
    if case["kind"] == "single":
        return X, y, [[stages[case["stage"]]]]
    return X, y, [candidates(stages[int(s)], d, local_search=case["tuned"], classification=case["problem"] == "class")
                  for s in case["stages"]]


def _batches(case, rounds):
    return [encode(r, tuned=case["kind"] == "single" or case["tuned"]) for r in rounds]


# -------------------------------------------------------------------- run --
_context = None


def _shared_context():
    """One context for the process, as a program keeps it: its stream, staging
    and scratch serve every dataset."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def prepare(case, seed):
    X, y, rounds = _problem(case, seed)
    if case["kind"] == "fit":
        import rils_rols_cpp
        model = rils_rols_cpp.rils_rols(case["problem"] == "class", case["calls"], 100, 0.001, 20, 1.0, False,
                                        seed % 100_000)
        model.set_precision(PRECISION[case["precision"]])
        return {"model": model, "X": X, "y": y}
    ctx = _shared_context()
    batches = _batches(case, rounds)
    # room for eight coefficients a tree, however many this seed's trees take
    room = 8 * case["trees"] if case["problem"] == "trees" else 1
    out = [(np.zeros(len(b), dtype=result_dtype()), np.zeros(max(room, b.n_coefs))) for b in batches]
    return {"ctx": ctx, "ds": ctx.dataset(X, y), "batches": batches, "out": out,
            "precision": PRECISION[case["precision"]]}


def run(state):
    if "model" in state:
        model, (n, d) = state["model"], state["X"].shape
        model.fit(state["X"], state["y"], n, d)
        return {"predicted": model.predict(state["X"], n, d), "fit_calls": model.get_fit_calls()}
    ds = state["ds"]
    state["ctx"].clear_column_cache()
    for batch, (res, coefs) in zip(state["batches"], state["out"]):
        ds.submit(batch, state["precision"], res, coefs)
        ds.wait()
    return [dict({k: res[k] for k in ("loss", "rmse", "size", "rank", "flags")},
                 **({"coefs": coefs} if batch.n_coefs else {}))
            for batch, (res, coefs) in zip(state["batches"], state["out"])]


# ------------------------------------------------------------------- work --
@functools.lru_cache(maxsize=64)
def _counted(key):
    case = dict(key)
    small = dict(case, n=64)
    _, _, rounds = _problem(small, 1)
    nodes = terms = cands = 0
    for b in _batches(case, rounds):
        cands += len(b)
        nodes += len(b.code)
        k = b.cands["n_factors"].astype(np.int64) + 1
        terms += int(np.sum(k * (k + 3))) if b.n_coefs else 2 * len(b)
    return cands, nodes, terms


def work(case):
    """Bytes: X and y read once, the results written once.  Flops: one
    operation per program word and row, and a least-squares refit of k terms
    as k (k + 3) per row (its k (k + 1) / 2 + k products and sums)."""
    n, d = case["n"], case["d"]
    if case["kind"] == "fit":
        return {"bytes": 8.0 * n * (2 * d + 2), "flops": 40.0 * n * case["calls"]}
    cands, nodes, terms = _counted(tuple(sorted(case.items())))
    return {"bytes": 8.0 * n * (d + 1) + 64.0 * cands, "flops": float(n) * (nodes + terms)}


# ------------------------------------------------------------------ exact --
_UNARY = {5: np.sin, 6: np.cos, 7: np.log, 8: np.exp, 9: np.sqrt, 10: np.square}
_BINARY = [np.add, np.subtract, np.multiply, np.divide, np.power, lambda a, b: (a < b) * 1.0,
           lambda a, b: (a == b) * 1.0, lambda a, b: (a != b) * 1.0, lambda a, b: np.where(a < b, a, b),
           lambda a, b: np.where(a > b, a, b)]


def _factors(batch):
    """Per candidate the factor programs as tuples of (opcode, operand), the
    constants by value."""
    out = []
    for c in batch.cands:
        progs, cur = [], []
        for w in batch.code[c["code_offset"]:c["code_offset"] + c["code_len"]].tolist():
            op, arg = w & 0xff, w >> 8
            if op == 11:
                progs.append(tuple(cur))
                cur = []
                continue
            const = op in (2, 4) or (op >= 16 and ((op - 16) & 7) >> 1 == 2)
            cur.append((op, float(batch.consts[arg]) if const else arg))
        out.append(progs)
    return out


def _column(prog, X):
    n, stack, t = len(X), [], None
    for op, arg in prog:
        if op in (1, 3):
            if op == 3:
                stack.append(t)
            t = X[:, arg]
        elif op in (2, 4):
            if op == 4:
                stack.append(t)
            t = np.full(n, arg)
        elif op in _UNARY:
            t = _UNARY[op](t)
        else:
            k = op - 16
            src = (k & 7) >> 1
            o = stack.pop() if src == 0 else (X[:, arg] if src == 1 else np.full(n, arg))
            t = _BINARY[k >> 3](t, o) if k & 1 else _BINARY[k >> 3](o, t)
    return np.asarray(t, dtype=np.float64)


def _refit(cols, y):
    """Rebuilt values of the least-squares refit on [cols, 1] by column-pivoted
    Householder QR (largest remaining norm first; a norm below eps of the
    largest ends the factorisation), terms below 1e-12 left out."""
    n = len(y)
    A = np.stack(cols + [np.ones(n), y])
    k = len(cols) + 1
    perm = list(range(k))
    first = None
    rank = size = min(n, k)
    for s in range(size):
        norms = np.sqrt(np.sum(A[perm[s:], s:] ** 2, axis=1))
        big = 0
        for j in range(1, len(norms)):  # a NaN wins only at the head
            if norms[j] > norms[big]:
                big = j
        first = norms[big] if s == 0 else first
        if norms[big] ** 2 < (first * np.finfo(float).eps) ** 2 / n * (n - s):
            rank = s
            break
        perm[s], perm[s + big] = perm[s + big], perm[s]
        v = A[perm[s], s:].copy()
        beta = -math.copysign(norms[big], v[0])
        v[0] -= beta
        rest = perm[s + 1:] + [k]
        w = (A[rest, s:] @ v) * (2.0 / (v @ v))
        A[rest, s:] -= w[:, None] * v
        A[perm[s], s] = beta
    c = np.array(A[k, :rank])
    for s in range(rank - 1, -1, -1):
        c[s] = c[s] / A[perm[s], s]
        c[:s] -= c[s] * A[perm[s], :s]
    yp = np.zeros(n)
    for s in range(rank):
        if not abs(c[s]) < 1e-12:
            f = cols[perm[s]] if perm[s] < k - 1 else 1.0
            yp = yp + (f if perm[s] < k - 1 and abs(c[s] - 1) < 1e-12 else c[s] * f)
    return yp


def exact(case, seed):
    """Loss and RMSE of every candidate.  None for a fit (what a search
    decides), for rounds that would take too long, and for the coefficients
    (those of a nearly rank-deficient design are not determined in 64 bits)."""
    if case["kind"] == "fit":
        return None
    cands, nodes, terms = _counted(tuple(sorted(case.items())))
    if case["n"] * (nodes * 2.0 + terms * 4.0) > 1.2e10:
        return None
    X, y, rounds = _problem(case, seed)
    X = np.asfortranarray(X)
    out = []
    with np.errstate(all="ignore"):
        sst = float(np.sum((y - np.mean(y)) ** 2))
        for b in _batches(case, rounds):
            seen, loss, rmse = {}, [], []
            for progs, cand in zip(_factors(b), b.cands):
                key = tuple(progs)
                if key not in seen:
                    cols = [_column(p, X) for p in progs]
                    yp = _refit(cols, y) if cand["mode"] else cols[0]
                    sse = float(np.sum((y - yp) ** 2))
                    r2, e = 1.0 - np.float64(sse) / sst, math.sqrt(sse / len(y)) if sse >= 0 else float("nan")
                    seen[key] = (1000.0, 1000.0) if r2 != r2 or e != e else (1.0 - r2, e)
                loss.append(seen[key][0])
                rmse.append(seen[key][1])
            out.append({"loss": np.array(loss), "rmse": np.array(rmse), "size": None, "rank": None, "flags": None,
                        "coefs": None})
    return out
