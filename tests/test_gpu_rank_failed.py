"""A failed candidate's segment of the rank sums: status 2 and four zero words
in the C interface's output, from the buckets and from the radix sort alike,
beside segments that have their sums."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [0, -1, 8])
@pytest.mark.parametrize("n", [2, 1000, 20011])
def test_failed_segments_have_zero_words(pkg, E, n, cap):
    dev = importlib.import_module("the-rule-and-compass_b200.device")
    rng = np.random.Generator(np.random.PCG64(n))
    x, y = rng.uniform(-1.0, 1.0, n), rng.normal(0, 1, n)
    x[-1] = -0.5
    ev = pkg.GpuEvaluator(x.astype(np.float32), n, 1, y.astype(np.float32))
    ev.set_fit_data(x, y)
    trees = [E.node(E.LOG, [E.constant(-1.0)]), E.input(0), E.node(E.LOG, [E.input(0)])]
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    ev.rank_tuning(cap, 0)
    prog, off, pcount, c0, nsets = ev._segments(prog, off, pcount, c0, kmax, 1)
    p = dev._p
    out = np.full((3, 4), 7, np.uint64)
    status, bb = np.zeros(3, np.int32), np.zeros(2, np.uint64)
    ms = dev.lib().rc_rank_score_batch(ev.ctx, p(prog, ctypes.c_uint32), p(off, ctypes.c_uint32),
                                       p(pcount, ctypes.c_int32), nsets, 1, kmax,
                                       p(c0, ctypes.c_double), p(out.reshape(-1), ctypes.c_uint64),
                                       p(status, ctypes.c_int32), p(bb, ctypes.c_uint64))
    assert ms >= 0 and status.tolist() == [2, 0, 2]
    assert not out[0].any() and not out[2].any()
    b = np.argsort(np.argsort(x)) * 2 + 1 - n  # distinct values
    assert int(out[1, 2]) == 0 and int(out[1, 3]) == int((b * b).sum())
    ev.close()
