"""The generation at the slot count from which the parents' metadata is read
back by itself (4,096): the oracle's children on both sides of it, and a pool
slot that is not a program fails the call there and leaves the pool usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALT = 255


def _setup(pkg, O, islands, pop):
    n = islands * pop
    words = O.random_arena(24, 2, 10, pkg.DEFAULT_VARIATION_OPS, 31, 3, n)
    err = np.array([((i * 7919) % 1009) / 1009.0 for i in range(n)], np.float64)
    x = np.linspace(-1, 1, 64, dtype=np.float32)
    ev = pkg.GpuEvaluator(np.stack([x, x * x]).reshape(-1), 64, 2, x)
    return ev, pkg.GenomePool(ev, islands, pop, 24), words, err


def _check(pkg, O, pool, words, err, islands, pop, **kw):
    pool.upload(0, words)
    dw, dl, dc, dh, de, _ = pool.vary(0, err, 1, 2, 10, 31, pkg.DEFAULT_VARIATION_OPS, **kw)
    rw, rl, rc, rh, re = O.next_generation(words, err, islands, pop, 24, 2, 10, 31, 1,
                                           pkg.DEFAULT_VARIATION_OPS, **kw)
    assert np.array_equal(dw, rw) and np.array_equal(dl, rl) and np.array_equal(dc, rc)
    assert np.array_equal(dh, rh) and np.array_equal(de.view(np.uint64), re.view(np.uint64))


@pytest.mark.parametrize("islands,pop", [(5, 819), (16, 256), (17, 241)])
def test_both_sides_of_the_line(pkg, O, islands, pop):
    ev, pool, words, err = _setup(pkg, O, islands, pop)
    _check(pkg, O, pool, words, err, islands, pop)
    _check(pkg, O, pool, words, err, islands, pop, restart=[1] + [0] * (islands - 1), dedup=False)
    ev.close()


@pytest.mark.parametrize("islands,pop", [(5, 819), (16, 256)])
def test_an_invalid_parent(pkg, O, islands, pop):
    ev, pool, words, err = _setup(pkg, O, islands, pop)
    bad = words.copy()
    bad[islands * pop - 1, :] = HALT
    bad[islands * pop - 1, 0] = 2  # ADD with an empty stack
    pool.upload(0, bad)
    with pytest.raises(pkg.DeviceError):
        pool.vary(0, err, 1, 2, 10, 31, pkg.DEFAULT_VARIATION_OPS)
    _check(pkg, O, pool, words, err, islands, pop)
    ev.close()
