"""Medians whose middle lies outside the sampled bracket: the rows that the
sample of a segment reads hold large residuals and all others small ones, so
the segment goes to the sort. The sort is seen to run (its launches), and the
values equal numpy's for segments sorted, settled by selection and failed,
alone and in one batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SAMPLES = 4096


def _sampled_rows(n, seg):
    """The rows whose keys are segment `seg`'s sample: the pair drawn from each
    of SAMPLES / 2 equal strata of the n / 2 pairs of rows."""
    u = lambda v: np.asarray(v, np.uint32)
    p = np.arange(SAMPLES // 2, dtype=np.uint32)
    h = u(seg * 0x9E3779B1 & 0xffffffff) ^ (p + u(0x7F4A7C15))
    h ^= h >> u(16)
    h *= u(0x85EBCA6B)
    h ^= h >> u(13)
    h *= u(0xC2B2AE35)
    h ^= h >> u(16)
    stride = n // 2 // (SAMPLES // 2)
    q = p.astype(np.int64) * stride + (h % u(stride)).astype(np.int64)
    return np.concatenate([2 * q, 2 * q + 1])


def _median(r):
    s = np.sort(np.abs(r))
    n = len(s)
    return s[n // 2] if n & 1 else 0.5 * (s[n // 2 - 1] + s[n // 2])


@pytest.mark.parametrize("large_sample", [True, False])
@pytest.mark.parametrize("n", [65538, 200003])
def test_misled_brackets(pkg, E, n, large_sample):
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.normal(0.0, 1.0, (3, n))
    for col, seg in ((0, 0), (1, 3)):
        far = np.zeros(n, bool)
        far[_sampled_rows(n, seg)] = True
        x[col, far if large_sample else ~far] += 1e6
    y = np.zeros(n)
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), n, 3, y.astype(np.float32))
    ev.set_fit_data(x.reshape(-1), y)
    failing = E.node(E.LOG, [E.constant(-1.0)])
    trees = {"a": E.input(0), "b": E.input(1), "c": E.input(2), "f": failing,
             "d": E.node(E.ADD, [E.input(2), E.constant(0.5)])}
    preds = {"a": x[0], "b": x[1], "c": x[2], "d": x[2] + 0.5}

    def run(names):
        """The kernels that the batch launched, its values checked."""
        plans = [pkg.gpu_fit_plan(trees[k], allow_no_constants=True) for k in names]
        prog, off, pcount, c0, _, kmax = pkg.pack_plans(plans)
        before = ev.launch_count()
        val, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, 0)
        assert status.tolist() == [2 if k == "f" else 0 for k in names]
        for k, v in zip(names, val):
            assert np.isnan(v) if k == "f" else v == _median(preds[k]), (names, k)
        return ev.launch_count() - before

    settled = run("ccfcd")
    first, both = run("acfcd"), run("acfbd")
    assert first > settled and both - settled == 2 * (first - settled)
    assert run("ccfbd") == first
    assert run("a") == first and run("c") == settled
    ev.close()
