"""Fits whose tiles run several chunks at once (small batches, grouped blocks)
against the same candidates in a batch large enough for one-group blocks and
several chains, and alone: the same bits, at row counts around a tile and
its chunks, for every arm with its own sweeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plans(pkg, E, metric):
    import importlib
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    if metric == 6:
        trees = [t for t in W.implicit_workload(24, 1, seed=5)[0] if t.constants()][:10]
    else:
        trees = W.fit_workload(10, 1, seed=8, nvars=4)[0]
    return [pkg.gpu_fit_plan(t) for t in trees]


@pytest.mark.parametrize("metric", [0, 1, 2, 4, 6])
@pytest.mark.parametrize("n", [1, 31, 2047, 2049, 4 * 2048 + 65])
def test_groups_and_chains_give_the_same_bits(pkg, E, metric, n):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.uniform(-2.0, 2.0, (4, n))
    y = 1.7 * np.exp(-0.5 * x[0] ** 2) + 0.4 * x[1] + rng.normal(0, 0.02, n)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 4, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    plans = _plans(pkg, E, metric)
    c, loss, status, _ = ev.fit_plans(plans, 6, metric)
    # repeated until the batch leaves the one-launch steps (8 items an SM)
    reps = 1 + (8 * 160) // (len(plans) * ((n + 2047) // 2048))
    big = ev.fit_plans(plans * reps, 6, metric)
    for r in (0, reps // 2, reps - 1):
        s = slice(r * len(plans), (r + 1) * len(plans))
        assert np.array_equal(big[0][s].view(np.uint64), c.view(np.uint64)), (metric, n, r)
        assert np.array_equal(big[1][s].view(np.uint64), loss.view(np.uint64))
        assert np.array_equal(big[2][s], status)
    for k in (0, 7):
        one = ev.fit_plans(plans[k:k + 1], 6, metric)
        m = plans[k].nconst
        assert np.array_equal(one[0][0, :m].view(np.uint64), c[k, :m].view(np.uint64)), (metric, n, k)
        assert one[1].view(np.uint64)[0] == loss.view(np.uint64)[k]
    ev.close()
