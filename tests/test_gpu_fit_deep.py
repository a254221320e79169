"""Fits of programs with many spill slots (right-nested sums, up to the 96
records of a plan), at the slot counts around what a 512-thread objective
block holds: accepted in every launch shape (alone, one small batch with
shallow programs, a large batch, the plain arm), with the same bits in all of
them, and solved."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2113  # a whole tile of 2,048 rows and a part of one


def _deep(E, slots):
    """x + (x + ( ... + (c * x))): that many spill slots."""
    t = E.node(E.MUL, [E.constant(0.5), E.input(0)])
    for k in range(slots - 1):
        t = E.node(E.ADD, [E.input(k % 3), t])
    return t


def _sum(x, slots):
    return sum(x[k % 3] for k in range(slots - 1))


def _evaluator(pkg, x, y):
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), x.shape[1], 3, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    return ev


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("slots", [27, 28, 29, 46])
def test_deep_fits(pkg, E, slots, metric):
    rng = np.random.Generator(np.random.PCG64(slots))
    x = rng.uniform(-1.0, 1.0, (3, N)).astype(np.float32).astype(np.float64)
    y = (_sum(x, slots) + 1.5 * x[0] + rng.normal(0, 0.01, N)).astype(np.float32).astype(np.float64)
    ev = _evaluator(pkg, x, y)
    deep = _deep(E, slots)
    shallow = E.node(E.ADD, [E.node(E.MUL, [E.constant(0.7), E.input(1)]), E.constant(0.1)])
    plans = [pkg.gpu_fit_plan(t) for t in (deep, shallow)]
    c, loss, status, _ = ev.fit_plans(plans, 6, metric)
    assert status.tolist() == [0, 0]
    if metric == 0:
        # linear in its one constant: the f32 sweeps' predictions (46 terms of
        # at most 1) are off by 46 * 46 * 2^-24 = 1.3e-4 at the very most, at
        # random by 2e-6 a row, which the 2,113 rows' mean divides by 40
        want = (x[0] @ (y - _sum(x, slots))) / (x[0] @ x[0])
        assert abs(c[0, 0] - want) <= 2e-6
    else:
        p = _sum(x, slots) + c[0, 0] * x[0]
        assert abs(loss[0] - (1.0 - abs(np.corrcoef(p, y)[0, 1]))) <= 1e-6
    bits = lambda a: np.ascontiguousarray(a).view(np.uint64)
    for k in (0, 1):
        m = plans[k].nconst
        one = ev.fit_plans(plans[k:k + 1], 6, metric)
        assert np.array_equal(bits(one[0][0, :m]), bits(c[k, :m])) and one[1][0] == loss[k]
        prog, off, pcount, c0, gauge, kmax = pkg.pack_plans(plans[k:k + 1])
        plain = ev.fit_batch_plain(prog, off, pcount, c0, gauge, kmax, 6, metric)
        assert np.array_equal(bits(plain[0][0, :m]), bits(c[k, :m])) and plain[1][0] == loss[k]
    # more (candidate, tile) items than the one-launch steps take
    reps = 1 + 8 * 160 // (2 * 2)
    big = ev.fit_plans(plans * reps, 6, metric)
    for r in (0, reps - 1):
        s = slice(2 * r, 2 * r + 2)
        assert np.array_equal(bits(big[0][s]), bits(c)) and np.array_equal(bits(big[1][s]), bits(loss))
        assert np.array_equal(big[2][s], status)
    ev.close()
