"""The median by selection (bracket from a sample, key lists, radix selection)
against numpy's sorted residuals, bit for bit where the prediction is exact:
row counts around the listed-everything bound, even and odd; ties (constant
residuals, two values, many equal keys across the middle), rows ordered so
that the sample misleads, and failing candidates. The same values as the sort
that the interquartile mean's path keeps (what = 1 is checked elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _median(r):
    s = np.sort(r)
    n = len(s)
    return s[n // 2] if n & 1 else 0.5 * (s[n // 2 - 1] + s[n // 2])


def _cases(n, rng):
    yield "normal", rng.standard_normal(n)
    yield "ties", np.round(rng.standard_normal(n) * 2.0)
    yield "constant", np.full(n, 0.25)
    two = np.where(np.arange(n) < n // 2, 1.0, 2.0)
    yield "two values", two
    yield "sorted rows", np.sort(rng.standard_cauchy(n))
    # every 64th pair of rows small: the strata see another middle than the rows
    odd = np.abs(rng.standard_normal(n)) + 10.0
    odd[: n // 2 + 3] *= 1e-12
    yield "binades", odd


@pytest.mark.parametrize("n", [1, 2, 3, 64, 1001, 32767, 32768, 32769, 65538, 200003])
def test_median_selection(pkg, E, n):
    rng = np.random.Generator(np.random.PCG64(n))
    trees = [E.input(0),                                        # |x - y| exactly rounded
             E.node(E.ADD, [E.input(0), E.constant(0.5)]),
             E.node(E.MUL, [E.constant(0.0), E.input(0)]),      # |0 - y|
             E.node(E.LOG, [E.constant(-1.0)]),                 # undefined
             E.node(E.NEG, [E.input(0)])]
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    for name, y in _cases(n, rng):
        x = rng.standard_normal(n)
        ev = pkg.GpuEvaluator(x.astype(np.float32), n, 1, y.astype(np.float32))
        ev.set_fit_data(x, y)
        val, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, 0)
        want = [_median(np.abs(x - y)), _median(np.abs((x + 0.5) - y)), _median(np.abs(0.0 * x - y)),
                None, _median(np.abs(-x - y))]
        assert status.tolist() == [0, 0, 0, 2, 0], (n, name)
        assert np.isnan(val[3])
        for k in (0, 1, 2, 4):
            assert val[k] == want[k], (n, name, k, val[k], want[k])
        ev.close()
