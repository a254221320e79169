"""The scorer's row tiles at the edges of their rule (about 32 tiles of 1,024
to 32,768 rows, chosen from n alone): values against the CPU reducer on the
device's own predictions or the f64 predictions, and the same bits for a
candidate alone and in its batch, with candidates that fail among them. The
two-pass correlation keeps a first-pass failure for its second pass."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 1025, 32768, 32769, 65537])
def test_scores_at_the_tile_edges(pkg, E, O, n):
    W = importlib.import_module("the-rule-and-compass_b200.workloads")
    trees, x, y = W.scoring_workload(20, n, seed=11, nvars=5)
    # fails in f32 alone (e^100 against its f64 value), in both, and late
    late = E.node(E.LOG, [E.node(E.ADD, [E.input(0), E.constant(float(-x[0].min()) * 0.999)])])
    trees += [E.node(E.EXP, [E.node(E.MUL, [E.constant(100.0), E.input(0)])]),
              E.node(E.SQRT, [E.input(1)]), late]
    prog, off = pkg.Population(trees).programs()
    ev = pkg.GpuEvaluator(x.reshape(-1), n, 5, y)
    preds = ev.predictions(prog, off).astype(np.float64)
    x64, y64 = x.astype(np.float64).reshape(-1), y.astype(np.float64)
    finite = 0
    for kind, tol in ((0, 1e-12), (4, 0.0), (5, 1e-9)):
        vals, status, _ = ev.score_batch(prog, off, kind)
        for k, t in enumerate(trees):
            t32 = t.clone()
            t32.set_constants([float(np.float32(c)) for c in t.constants()])
            want64 = O.score_pred(O.predict(t32, x64, n, 5), y64, kind, 0)
            want32 = O.score_pred(preds[k], y64, kind, 0)
            if not np.isfinite(want64):
                assert status[k] == 2 and np.isinf(vals[k]), (n, kind, k)
                continue
            if status[k] == 0:
                finite += 1
                bound = tol * (1.0 + abs(want64))
                assert min(abs(vals[k] - want32), abs(vals[k] - want64)) <= bound or \
                    abs(vals[k] - want64) <= 1e-9 * abs(want64), (n, kind, k, vals[k], want64)
            p1 = prog[off[k]:off[k + 1]]
            one, st1, _ = ev.score_batch(p1, np.array([0, len(p1)], np.uint32), kind)
            assert st1[0] == status[k]
            assert one.view(np.uint64)[0] == vals[k:k + 1].view(np.uint64)[0], (n, kind, k)
    assert finite >= 12
    ev.close()
