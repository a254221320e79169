"""A fit's captured graph is replayed only for the buffers that it was captured
with: row weights and label signs set, replaced and cleared between fits of
one shape, and batches of one shape whose tables lie at other offsets. Every
result equals that of a context that made no fit before, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2113


def _rows():
    rng = np.random.Generator(np.random.PCG64(11))
    x = rng.uniform(-1.0, 1.0, (2, N))
    y = np.sin(1.3 * x[0]) + 0.4 * x[1] + rng.normal(0, 0.05, N)
    return x, y, rng.uniform(0.1, 2.0, N)


def _evaluator(pkg, x, y, w=None):
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), N, 2, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y, w)
    return ev


def _fit(ev, plans, metric=0):
    c, loss, status, _ = ev.fit_plans(plans, 6, metric)
    return c.tobytes(), loss.tobytes(), status.tobytes()


def _trees(E):
    wave = E.node(E.SIN, [E.node(E.MUL, [E.constant(1.0), E.input(0)])])
    return [E.node(E.ADD, [wave, E.node(E.MUL, [E.constant(0.5), E.input(1)])]),
            E.node(E.ADD, [E.node(E.MUL, [E.constant(0.2), E.input(0)]), E.constant(0.1)])]


def _fresh(pkg, plans, x, y, w=None, sign=None, metric=0):
    ev = _evaluator(pkg, x, y, w)
    if sign is not None:
        ev.set_fit_sign(sign)
    out = _fit(ev, plans, metric)
    ev.close()
    return out


def test_weights_between_fits(pkg, E):
    x, y, w = _rows()
    plans = [pkg.gpu_fit_plan(t) for t in _trees(E)]
    plain, weighted = _fresh(pkg, plans, x, y), _fresh(pkg, plans, x, y, w)
    assert plain != weighted
    ev = _evaluator(pkg, x, y)
    for want, change in ((plain, lambda: None),
                         (weighted, lambda: ev.set_score_weights(w)),
                         (plain, lambda: ev.set_score_weights(None)),
                         (weighted, lambda: ev.set_fit_data(x.reshape(-1), y, w)),
                         (_fresh(pkg, plans, x, y, 3.0 * w), lambda: ev.set_score_weights(3.0 * w)),
                         (plain, lambda: ev.set_fit_data(x.reshape(-1), y))):
        change()
        for _ in range(3):  # direct, captured, replayed
            assert _fit(ev, plans) == want
    ev.close()


def test_signs_between_fits(pkg, E):
    x, y, _ = _rows()
    plans = [pkg.gpu_fit_plan(t) for t in _trees(E)]
    up = np.where(x[0] + 0.3 * np.sin(40.0 * x[1]) > 0, 1.0, -1.0)
    ev = _evaluator(pkg, x, y)
    for sign in (up, -up, np.where(x[1] > 0.2, 1.0, -1.0)):
        ev.set_fit_sign(None)
        ev.set_fit_sign(sign)
        want = _fresh(pkg, plans, x, y, sign=sign, metric=3)
        for _ in range(3):
            assert _fit(ev, plans, 3) == want
    ev.close()


def test_tables_at_other_offsets(pkg, E):
    """(x + c) + x has one record more than -(c * x), and one instruction pair
    fewer: batches of as many of both in other shares are of one size in all,
    with their instruction tables 512 bytes apart."""
    x, y, _ = _rows()
    add = E.node(E.ADD, [E.node(E.ADD, [E.input(0), E.constant(0.5)]), E.input(1)])
    neg = E.node(E.NEG, [E.node(E.MUL, [E.constant(0.5), E.input(0)])])
    plans = [pkg.gpu_fit_plan(t) for t in (_trees(E)[0], add, neg)]
    one = [plans[:1] + plans[1:2] * k + plans[2:3] * (64 - k) for k in (48, 16)]
    want = [_fresh(pkg, p, x, y) for p in one]
    ev = _evaluator(pkg, x, y)
    for k in (0, 0, 0, 1, 1, 1, 0, 1):
        assert _fit(ev, one[k]) == want[k]
    ev.close()
