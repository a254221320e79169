"""The implicit score at row counts that end inside a warp's group of rows: a
warp whose last lanes had no rows used to wait at its vote for lanes that had
left the loop, so the call never returned. Values against the oracle (f32
rows, f64 sums: 1e-4 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 65, 250, 257, 16383, 16384 + 30])
def test_implicit_score_ragged_rows(pkg, E, O, n):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.uniform(0.3, 1.0, (2, n)).astype(np.float32).astype(np.float64)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 2, np.zeros(n, np.float32))
    ev.set_fit_data(x.reshape(-1), np.zeros(n))
    trees = [E.node(E.SUB, [E.node(E.ADD, [E.node(E.SQUARE, [E.input(0)]),
                                           E.node(E.SQUARE, [E.input(1)])]), E.constant(1.5)]),
             E.node(E.MUL, [E.node(E.SIN, [E.input(0)]), E.input(1)]),
             E.node(E.LOG, [E.node(E.SUB, [E.input(0), E.constant(5.0)])])]  # undefined
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    val, status, _ = ev.implicit_score(prog, off, pcount, c0, kmax)
    assert status.tolist() == [0, 0, 2]
    for k in (0, 1):
        want = O.implicit_score(trees[k], x.reshape(-1), n, 2)
        assert abs(val[k] - want) <= 1e-4 * (1 + abs(want)), (n, k)
    ev.close()
