"""Work items of several row tiles (batches with items to spare): every program
has the bits, status and predictions that it has alone, where an item is one
tile, at row counts that end inside a span and inside a tile, for both kernel
shapes, with candidates that fail in the first, a middle or only the last row,
and in f32 alone."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COPIES = 4200  # spans of two tiles and more from 9 tiles on


def _programs(E, x, deep):
    c, v = E.constant, E.input
    at = lambda r: float(np.float32(x[0, r]) * np.float32(0.9999))  # noqa: E731
    n = x.shape[1]
    out = [E.node(E.MUL, [v(0), E.node(E.SIN, [v(1)])]), E.node(E.SUB, [v(2), c(0.25)]),
           # x0 falls from 2 to 1: undefined from a middle row on, in the last row alone
           E.node(E.LOG, [E.node(E.SUB, [v(0), c(at(n // 2))])]),
           E.node(E.LOG, [E.node(E.SUB, [v(0), c(float(np.float32(x[0, n - 2] + x[0, n - 1]) / 2))])]),
           E.node(E.LOG, [E.node(E.NEG, [v(0)])]),                       # in every row
           E.node(E.DIV, [E.node(E.EXP, [E.node(E.MUL, [c(60.0), v(0)])]), c(1e30)])]  # f32 overflow
    if deep:  # more spill slots than the shallow shape keeps
        def wrap(t):
            for k in range(8):
                t = E.node(E.ADD, [E.node(E.MUL, [v(k % 3), v((k + 1) % 3)]), t])
            return t
        spine = v(1)
        for k in range(12):
            spine = E.node(E.ADD, [v(k % 3), spine])
        out = [E.node(E.ADD, [spine, wrap(t)]) for t in out]
    return out


def _data(n):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.normal(0.0, 1.0, (3, n)).astype(np.float32)
    x[0] = np.linspace(2.0, 1.0, n, dtype=np.float32)
    y = (np.sin(x[1]) + 0.1 * x[2]).astype(np.float32)
    return x, y


@pytest.mark.parametrize("n", [8193, 33001, 65537])
@pytest.mark.parametrize("kind,deep", [(0, False), (1, False), (2, False), (4, False), (5, False),
                                       (10, False), (0, True), (4, True)])
def test_spans_give_the_bits_of_single_tiles(pkg, E, n, kind, deep):
    x, y = _data(n)
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, y)
    if kind == 10:
        ev.set_fit_sign(np.where(y > 0, 1.0, -1.0))
        ev.set_score_weights(np.where(np.arange(n) % 7 == 0, 0.0, 1.5))
    trees = _programs(E, x, deep)
    reps = COPIES // len(trees)
    prog, off = pkg.Population(trees * reps).programs()
    vals, status, _ = ev.score_batch(prog, off, kind)
    ok = 0
    for k in range(len(trees)):
        p1 = prog[off[k]:off[k + 1]]
        one, st1, _ = ev.score_batch(p1, np.array([0, len(p1)], np.uint32), kind)
        ok += st1[0] == 0
        assert (status[k::len(trees)] == st1[0]).all(), (n, kind, k)
        assert (vals[k::len(trees)].view(np.uint64) == one.view(np.uint64)[0]).all(), (n, kind, k)
    assert ok >= 2
    ev.close()


def test_predictions_over_spans(pkg, E):
    n = 8193
    x, y = _data(n)
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 3, y)
    trees = _programs(E, x, False)
    prog, off = pkg.Population(trees * (COPIES // len(trees))).programs()
    big = ev.predictions(prog, off)
    small = ev.predictions(prog[:off[len(trees)]], off[:len(trees) + 1])
    for k in range(len(big)):
        assert np.array_equal(big[k].view(np.uint32), small[k % len(trees)].view(np.uint32)), k
    ev.close()
