"""Folded constant subtrees and shared columns of the scorer at the row counts
that they start from (393,216, a correlation 131,072): a batch just past them,
and one just below, gives every program the bits and status it gets alone
(where nothing is folded or shared), in scores and in predictions."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _programs(pkg, E, rng, count):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    c, x = E.constant, E.input
    cc = lambda: E.node(E.MUL, [E.node(E.SIN, [c(float(rng.uniform(-2, 2)))]), c(1.5)])  # noqa: E731
    out = [E.node(E.ADD, [cc(), x(0)]), E.node(E.MUL, [E.node(E.EXP, [x(1)]), cc()]),
           E.node(E.DIV, [cc(), E.node(E.COS, [x(2)])]), E.node(E.IF, [x(0), cc(), E.node(E.SIN, [x(1)])]),
           E.node(E.LOG, [cc()]), E.node(E.LOG, [c(-1.0)]), E.node(E.EXP, [E.node(E.EXP, [c(9.0)])]),
           E.node(E.EXP, [E.node(E.MUL, [c(40.0), x(0)])]), E.node(E.SIN, [x(0)]),
           E.node(E.ADD, [E.node(E.SIN, [x(0)]), E.node(E.EXP, [x(0)])]), c(2.0)]
    t = E.node(E.SIN, [x(1)])  # a deep right spine, constants and columns at every level
    for k in range(20):
        t = E.node(E.ADD, [E.node(E.MUL, [cc(), E.node(E.COS, [x(k % 3)])]), t])
    out.append(t)
    return out + [W.random_scoring_tree(rng, 3) for _ in range(count - len(out))]


@pytest.mark.parametrize("kind,n,count", [(0, 393216, 44), (1, 393253, 44), (4, 393253, 44),
                                          (10, 393216, 44), (0, 393215, 44), (5, 131072, 132),
                                          (6, 131077, 132), (5, 131071, 132)])
def test_a_batch_past_the_line_gives_the_bits_of_each_program_alone(pkg, E, kind, n, count):
    rng = np.random.Generator(np.random.PCG64(n + kind))
    x = rng.normal(0.0, 1.0, (3, n)).astype(np.float32)
    y = (x[0] * x[1] + np.sin(x[2])).astype(np.float32)
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, y)
    if kind == 10:
        ev.set_fit_sign(np.where(y > 0, 1.0, -1.0))
    prog, off = pkg.Population(_programs(pkg, E, rng, count)).programs()
    vals, status, _ = ev.score_batch(prog, off, kind)
    for k in range(count):
        p1 = prog[off[k]:off[k + 1]]
        one, st1, _ = ev.score_batch(p1, np.array([0, len(p1)], np.uint32), kind)
        assert status[k] == st1[0], (kind, n, k)
        assert vals[k:k + 1].view(np.uint64)[0] == one.view(np.uint64)[0], (kind, n, k)
    ev.close()


def test_predictions_past_the_line(pkg, E):
    n = 393221
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.normal(0.0, 1.0, (3, n)).astype(np.float32)
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, x[0])
    prog, off = pkg.Population(_programs(pkg, E, rng, 44)).programs()
    big = ev.predictions(prog, off)
    for k in range(44):
        p1 = prog[off[k]:off[k + 1]]
        one = ev.predictions(p1, np.array([0, len(p1)], np.uint32))[0]
        ok = ~np.isnan(one)
        assert np.array_equal(np.isnan(big[k]), ~ok), k
        assert np.array_equal(big[k][ok].view(np.uint32), one[ok].view(np.uint32)), k
    ev.close()
