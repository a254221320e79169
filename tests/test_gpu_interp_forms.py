"""The device words of the fit interpreter over every operand form: each
binary operator with a constant, an input, a constant-free subtree and a
subtree holding a constant on either side, and each unary operator over the
two kinds of subtree, inside a sum that makes the whole expression an operand
of a live operator. Constant adjoints (the assembly's forward and reverse
sweeps) against the oracle's backward pass, f32 against f64 at 4 ulp per
operator on values of order one (1e-4 relative), and the implicit score (the
input-mode sweeps) against the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(E):
    c, x = E.constant, E.input
    kids = {"const": lambda: c(1.3), "input": lambda: x(0),
            "free": lambda: E.node(E.ADD, [E.node(E.SQUARE, [x(1)]), x(0)]),
            "live": lambda: E.node(E.ADD, [E.node(E.MUL, [c(0.7), x(1)]), c(0.9)])}
    out = []
    for op in (E.ADD, E.SUB, E.MUL, E.DIV, E.POW):
        for a in kids:
            for b in kids:
                out.append(E.node(op, [kids[a](), kids[b]()]))
    for op in (E.NEG, E.SQUARE, E.SIN, E.COS, E.EXP, E.TANH, E.SIG, E.GAUSS, E.LOG, E.SQRT, E.ABS,
               E.CUBE, E.SINH, E.COSH, E.ERF, E.ERFC, E.TAN):
        for k in ("free", "live"):
            out.append(E.node(op, [kids[k]()]))
    # an operand of a live operator on either side, and alone under it
    trees = []
    for i, t in enumerate(out):
        outer = [E.ADD, E.SUB, E.MUL][i % 3]
        other = E.node(E.MUL, [c(1.1), E.node(E.SIN, [x(1)])])
        trees.append(E.node(outer, [t.clone(), other.clone()]))
        trees.append(E.node(outer, [other, t]))
    return trees


def test_constant_adjoints_of_every_form(pkg, E, O):
    n = 70
    rng = np.random.Generator(np.random.PCG64(3))
    x = rng.uniform(0.3, 1.0, (2, n)).astype(np.float32).astype(np.float64)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 2, np.zeros(n, np.float32))
    ev.set_fit_data(x.reshape(-1), np.zeros(n))
    trees = _forms(E)
    plans = [pkg.gpu_fit_plan(t) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    val, g = ev.grad_batch(prog, off, pcount, c0, kmax, 1, 3, 64)
    for k, t in enumerate(trees):
        for r in (0, 1, 31, 63):
            v, cg, _ = O.row_grad(t, x[:, 3 + r])
            assert abs(val[k, r] - v) <= 1e-4 * (1 + abs(v)), (k, t)
            scale = 1 + np.abs(cg).max()
            assert np.all(np.abs(g[k, r, :plans[k].nconst] - cg) <= 1e-4 * scale), (k, t)
    ev.close()


def test_implicit_score_of_every_form(pkg, E, O):
    n = 128
    rng = np.random.Generator(np.random.PCG64(4))
    x = rng.uniform(0.3, 1.0, (2, n)).astype(np.float32).astype(np.float64)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 2, np.zeros(n, np.float32))
    ev.set_fit_data(x.reshape(-1), np.zeros(n))
    trees = _forms(E)
    plans = [pkg.gpu_fit_plan(t) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    val, status, _ = ev.implicit_score(prog, off, pcount, c0, kmax)
    finite = 0
    for k, t in enumerate(trees):
        want = O.implicit_score(t, x.reshape(-1), n, 2)
        if not np.isfinite(want):
            assert status[k] == 2
            continue
        assert status[k] == 0
        assert abs(val[k] - want) <= 1e-4 * (1 + abs(want)), (k, t, val[k], want)
        finite += 1
    assert finite > 100
    ev.close()
