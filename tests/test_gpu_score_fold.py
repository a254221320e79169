"""Folded constant subtrees and shared columns of the scorer: a batch large
enough for them gives every program the bits it gets alone (where nothing is
folded or shared), for programs made of every constant form (on either side,
nested, through IF, undefined, overflowing) and sin / cos / exp of inputs at
every depth, in values, statuses and raw predictions, on both kernel shapes
and through the f64 lane."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _programs(E, rng):
    c, x = E.constant, E.input
    cc = lambda: E.node(E.MUL, [E.node(E.SIN, [c(float(rng.uniform(-2, 2)))]), c(1.5)])  # noqa: E731
    out = [E.node(E.ADD, [cc(), x(0)]), E.node(E.ADD, [x(0), cc()]), E.node(E.SUB, [cc(), cc()]),
           E.node(E.MUL, [E.node(E.EXP, [x(1)]), cc()]), E.node(E.DIV, [cc(), E.node(E.COS, [x(2)])]),
           E.node(E.IF, [cc(), x(0), x(1)]), E.node(E.IF, [x(0), cc(), E.node(E.SIN, [x(1)])]),
           E.node(E.IF, [cc(), cc(), cc()]), E.node(E.LOG, [cc()]), E.node(E.LOG, [c(-1.0)]),
           E.node(E.EXP, [E.node(E.EXP, [c(9.0)])]), E.node(E.EXP, [E.node(E.MUL, [c(40.0), x(0)])]),
           E.node(E.MIN, [x(0), E.node(E.DIV, [c(1.0), E.node(E.EXP, [E.node(E.EXP, [c(9.0)])])])]),
           E.node(E.NEG, [cc()]), E.node(E.SIN, [x(0)]), E.node(E.COS, [E.node(E.COS, [x(0)])]),
           E.node(E.POW, [E.node(E.SQUARE, [x(0)]), cc()]), E.node(E.SQRT, [cc()]), c(2.0),
           E.node(E.ADD, [E.node(E.SIN, [x(0)]), E.node(E.EXP, [x(0)])])]
    # deep right spine with constants and columns at every level (20 entries)
    t = E.node(E.SIN, [x(1)])
    for k in range(20):
        t = E.node(E.ADD, [E.node(E.MUL, [cc(), E.node(E.COS, [x(k % 3)])]), t])
    out.append(t)
    return out


@pytest.mark.parametrize("kind", [0, 2, 4, 5])
def test_a_large_batch_gives_the_bits_of_each_program_alone(pkg, E, kind):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    rng = np.random.Generator(np.random.PCG64(12))
    n = 16384 + 37
    x, y = W.scoring_data(n, 9, 3)
    trees = _programs(E, rng) + [W.random_scoring_tree(rng, 3) for _ in range(40)]
    reps = 1 + (1 << 24) // (n * len(trees))
    prog, off = pkg.Population(trees * reps).programs()
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, y)
    vals, status, _ = ev.score_batch(prog, off, kind)
    for k in range(len(trees)):
        p1 = prog[off[k]:off[k + 1]]
        one, st1, _ = ev.score_batch(p1, np.array([0, len(p1)], np.uint32), kind)
        for j in (k, k + len(trees) * (reps - 1)):
            assert status[j] == st1[0], (kind, k)
            assert vals[j:j + 1].view(np.uint64)[0] == one.view(np.uint64)[0], (kind, k, vals[j], one)
    ev.close()


def test_predictions_of_a_large_batch(pkg, E):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    rng = np.random.Generator(np.random.PCG64(13))
    n = 65536 + 5
    x, y = W.scoring_data(n, 9, 3)
    trees = _programs(E, rng) * 13
    prog, off = pkg.Population(trees).programs()
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, y)
    big = ev.predictions(prog, off)
    for k in range(len(trees) // 13):
        p1 = prog[off[k]:off[k + 1]]
        one = ev.predictions(p1, np.array([0, len(p1)], np.uint32))
        a, b = big[k], one[0]
        assert np.array_equal(np.isnan(a), np.isnan(b)), k
        ok = ~np.isnan(a)
        assert np.array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32)), k
    ev.close()
