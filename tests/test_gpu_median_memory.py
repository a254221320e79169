"""Device memory that a batch of medians reserves: the listed keys, and above
the listed-everything bound the samples that the bracket reads, with the
reservation's own quarter of headroom; not more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,segs", [(1000, 5000), (32768, 600), (32769, 600)])
def test_reservation(pkg, E, n, segs):
    rng = np.random.Generator(np.random.PCG64(n))
    x, y = rng.normal(0, 1, n), rng.normal(0, 1, n)
    ev = pkg.GpuEvaluator(x.astype(np.float32), n, 1, y.astype(np.float32))
    ev.set_fit_data(x, y)
    plans = [pkg.gpu_fit_plan(E.node(E.ADD, [E.input(0), E.constant(k / 256.0)])) for k in range(segs)]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    val, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, 0)
    assert not status.any()
    for k in (0, segs - 1):
        s = np.sort(np.abs((x + k / 256.0) - y))
        assert val[k] == (s[n // 2] if n & 1 else 0.5 * (s[n // 2 - 1] + s[n // 2]))
    keys = 8 * (n + (0 if n <= 32768 else 4096))
    # a program of 3 records: under 1 KB of lists, tables and outputs a segment
    assert ev.arena_report().fs_dev_bytes <= 1.25 * (segs * (keys + 1024) + (1 << 20))
    ev.close()
