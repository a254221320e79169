"""Counts of the tiles that lost trials' objective sweeps leave out: none in a
table of one tile (the sum so far is then empty), never a sweep's first tile,
some where trials are rejected over many tiles; results do not depend on
them."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(pkg, n, plans, metric):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.uniform(-2.0, 2.0, (4, n))
    y = 1.7 * np.exp(-0.5 * x[0] ** 2) * np.cos(2.3 * x[1]) + 0.4 * x[2] + rng.normal(0, 0.05, n)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 4, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    res = [ev.fit_plans(plans, 12, metric) for _ in range(2)]
    assert all(a.tobytes() == b.tobytes() for a, b in zip(res[0][:3], res[1][:3]))
    out = ev.fit_sweeps(len(plans)), ev.fit_lost_tiles(len(plans))
    with pytest.raises(pkg.DeviceError):
        ev.fit_lost_tiles(len(plans) + 1)
    ev.close()
    return out


@pytest.mark.parametrize("metric", [0, 2, 4, 6])
def test_counts(pkg, metric):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    if metric == 6:
        trees = [t for t in W.implicit_workload(24, 1, seed=5)[0] if t.constants()][:12]
    else:
        trees = W.fit_workload(48, 1, seed=8, nvars=4)[0]
    plans = [pkg.gpu_fit_plan(t) for t in trees]
    _, lost = _fit(pkg, 2048, plans, metric)
    assert not lost.any()
    n = 40 * 2048 + 5
    sweeps, lost = _fit(pkg, n, plans, metric)
    assert (lost >= 0).all() and (lost <= 40 * sweeps[:, [1, 3]]).all()
    if metric in (0, 4):
        assert lost[:, 0].sum() > 0
    if metric == 2:  # its trials are correlations: no sum to exceed
        assert not lost.any()
