"""Weighted fits in one-launch batches (several chunks of a tile at once) and in
batches large enough for one-group blocks and chains: the same bits, row
weights of every size and zero among them, for each arm that sums weighted
terms."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [33, 2049, 4 * 2048 + 65])
def test_weighted_groups_give_the_same_bits(pkg, metric, n):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    rng = np.random.Generator(np.random.PCG64(100 + n))
    x = rng.uniform(-2.0, 2.0, (4, n))
    y = 1.7 * np.exp(-0.5 * x[0] ** 2) + 0.4 * x[1] + rng.normal(0, 0.02, n)
    w = rng.uniform(0.0, 3.0, n)
    w[rng.random(n) < 0.1] = 0.0
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 4, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y, w)
    ev.set_fit_sign(np.where(y > 0.7, 1.0, -1.0))
    plans = [pkg.gpu_fit_plan(t) for t in W.fit_workload(10, 1, seed=8, nvars=4)[0]]
    c, loss, status, _ = ev.fit_plans(plans, 6, metric)
    assert (status == 0).any()
    reps = 1 + (8 * 160) // (len(plans) * ((n + 2047) // 2048))
    big = ev.fit_plans(plans * reps, 6, metric)
    for r in (0, reps - 1):
        s = slice(r * len(plans), (r + 1) * len(plans))
        assert np.array_equal(big[0][s].view(np.uint64), c.view(np.uint64)), (metric, n, r)
        assert np.array_equal(big[1][s].view(np.uint64), loss.view(np.uint64))
        assert np.array_equal(big[2][s], status)
    ev.close()
