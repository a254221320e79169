"""Rank sums, medians and interquartile means of batches whose deepest program
(a right-nested sum, up to the 96 records of a plan) has more spill slots than
a four-row key sweep holds: accepted, and equal to numpy's on predictions
that are exact in f64, for the deep and the shallow programs of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _deep(E, slots):
    """x0 + (x1 + (x2 + (x0 + ... + (2 * x0)))): that many spill slots."""
    t = E.node(E.MUL, [E.constant(2.0), E.input(0)])
    for k in range(slots - 1):
        t = E.node(E.ADD, [E.input(k % 3), t])
    return t


def _centred(a):
    """2 * (midrank - mean midrank), whole numbers: first + past-last position - n."""
    s = np.sort(a)
    return np.searchsorted(s, a, "left") + np.searchsorted(s, a, "right") - len(a)


@pytest.mark.parametrize("radix", [False, True])
@pytest.mark.parametrize("n", [3, 1025, 9001, 70003])
@pytest.mark.parametrize("slots", [27, 28, 29, 46])
def test_deep_statistics(pkg, E, slots, n, radix):
    rng = np.random.Generator(np.random.PCG64(1000 * slots + n))
    # eighths up to 512: every sum below is exact
    x = rng.integers(-4096, 4097, (3, n)) / 8.0
    y = rng.integers(-4096, 4097, n) / 8.0
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 3, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    trees = [E.input(1), _deep(E, slots), E.node(E.NEG, [E.input(2)])]
    preds = [x[1], sum(x[k % 3] for k in range(slots - 1)) + 2.0 * x[0], -x[2]]
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    ev.rank_tuning(-1 if radix else 0, 0)
    sums, status, bb, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
    b = _centred(y)
    assert status.tolist() == [0, 0, 0] and bb == int(b @ b)
    for k, p in enumerate(preds):
        a = _centred(p)
        assert sums[k] == (int(a @ b), int(a @ a)), (slots, n, k)
    if radix:
        ev.close()
        return
    for what in (0, 1):
        val, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, what)
        assert status.tolist() == [0, 0, 0]
        for k, p in enumerate(preds):
            s = np.sort(np.abs(p - y))
            lo, hi = (0, n) if n < 4 else (n // 4, 3 * n // 4)
            # (sums of eighths below 2^53 are exact; one division)
            want = (s[n // 2] if n & 1 else 0.5 * (s[n // 2 - 1] + s[n // 2])) if what == 0 else \
                s[lo:hi].sum() / (hi - lo)
            assert val[k] == want, (slots, n, k, what)
    ev.close()


@pytest.mark.parametrize("n", [9001, 70003])
def test_wide_batches(pkg, E, n):
    """More than eight key blocks an SM: a sort's keys two rows a thread."""
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.integers(-4096, 4097, (3, n)) / 8.0
    y = rng.integers(-4096, 4097, n) / 8.0
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 3, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    trees = [E.input(1), _deep(E, 5), E.node(E.LOG, [E.constant(-1.0)])]
    preds = [x[1], sum(x[k % 3] for k in range(4)) + 2.0 * x[0], None]
    reps = 1 + 8 * 160 // (3 * ((n + 8191) // 8192))
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees] * reps
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    lo, hi = n // 4, 3 * n // 4
    val, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, 1)
    assert status.tolist() == [0, 0, 2] * reps
    for k in (0, 1):
        s = np.sort(np.abs(preds[k] - y))
        assert (val[k::3] == s[lo:hi].sum() / (hi - lo)).all(), (n, k)
    ev.rank_tuning(-1, 0)
    sums, status, _, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
    b = _centred(y)
    for k in (0, 1):
        a = _centred(preds[k])
        assert set(sums[k::3]) == {(int(a @ b), int(a @ a))}, (n, k)
    ev.close()
