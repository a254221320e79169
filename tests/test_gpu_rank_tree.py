"""The bucketed rank sums against the radix sort's where the splitters' search
tree changes its depth: row counts that give one splitter fewer, as many and
one more than a power of two, and columns of one to nine values (as few
splitters, all of them with equality buckets), and samples of 1 to 16 keys a
sorting thread. Whole numbers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8193, 14336, 16384, 16385, 32769, 34817, 131073, 300007, 700001, 2097152,
                               2099201])
def test_bucketed_sums_equal_the_sorted_ones(pkg, E, n):
    rng = np.random.Generator(np.random.PCG64(n))
    cols = np.stack([rng.standard_normal(n)] +
                    [rng.integers(0, k, n) * 0.375 - 1.0 for k in (2, 3, 4, 5, 8, 9)])
    y = np.round(rng.standard_normal(n), 2)
    ev = pkg.GpuEvaluator(cols.astype(np.float32).reshape(-1), n, len(cols), y.astype(np.float32))
    ev.set_fit_data(cols.reshape(-1), y)
    trees = [E.node(E.ADD, [E.input(v), E.constant(0.5)]) for v in range(len(cols))]
    trees.append(E.node(E.MUL, [E.constant(0.0), E.input(1)]))
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    sums, status, _, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
    assert list(status) == [0] * len(trees) and ev.rank_fallbacks() == 0
    ev.rank_tuning(-1, 0)
    want, status, _, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
    assert ev.rank_fallbacks() == len(trees)
    assert sums == want
    ev.close()


@pytest.mark.parametrize("n,values", [(20001, 2000), (65536, 20000), (300007, 6000), (300007, 150000)])
def test_groups_of_ties_equal_the_sorted_ones(pkg, E, n, values):
    """Digit groups of equal keys, of a few distinct ones and of both, and
    buckets of more keys than the block holds in registers; a comparison bound
    of one sorts every bucket with a mixed group."""
    rng = np.random.Generator(np.random.PCG64(values))
    x = rng.integers(0, values, n) / 64.0
    x[: n // 3] = x[: n // 3] % 8.0  # a third of the rows in few buckets
    y = np.round(rng.standard_normal(n), 3)
    ev = pkg.GpuEvaluator(x.astype(np.float32), n, 1, y.astype(np.float32))
    ev.set_fit_data(x, y)
    trees = [E.node(E.ADD, [E.node(E.MUL, [E.constant(c), E.input(0)]), E.constant(1.0)])
             for c in (1.0, -0.3)]
    plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in trees]
    prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
    got = []
    for cap, gmax in ((0, 0), (0, 1), (-1, 0)):
        ev.rank_tuning(cap, gmax)
        sums, status, _, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
        assert list(status) == [0, 0]
        got.append(sums)
    assert got[0] == got[2] and got[1] == got[2]
    ev.close()
