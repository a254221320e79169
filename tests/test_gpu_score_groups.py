"""Scores do not depend on the candidates of a work item: every group size of
the tuning file, for both kernel shapes (the 64-thread one has fewer threads
than a group of 32 has partial sums), in batches large enough to keep it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1100  # two tiles


def _trees(E, deep):
    v, c = E.input, E.constant
    out = []
    for k in range(40):
        t = E.node(E.MUL, [v(k % 3), c(0.25 + k / 16.0)])
        for j in range(18 if deep else 2):  # more than 15 spill slots: the 64-thread shape
            t = E.node(E.ADD, [v((j + k) % 3), t])
        out.append(t)
    out[7] = E.node(E.ADD, [out[7], E.node(E.LOG, [c(-1.0)])])
    return out


@pytest.mark.parametrize("deep", [False, True])
@pytest.mark.parametrize("group", [1, 8, 16, 32])
def test_every_group_size_gives_the_same_bits(pkg, E, tmp_path, deep, group):
    rng = np.random.Generator(np.random.PCG64(4))
    x = rng.normal(0.0, 1.0, (3, N)).astype(np.float32)
    y = (x[0] - x[1]).astype(np.float32)
    trees = _trees(E, deep)
    # 32-program groups x two tiles: 16 items an SM and more
    reps = 1 + 32 * 16 * 160 // (2 * len(trees))
    prog, off = pkg.Population(trees * reps).programs()
    ev = pkg.GpuEvaluator(x.reshape(-1), N, 3, y)
    alone, st1, _ = ev.score_batch(prog[:off[len(trees)]], off[:len(trees) + 1], 0)
    path = tmp_path / "tune"
    path.write_text(f"{N} 3 0 {group}\n{N} 3 1 {group}\n")
    assert ev.autotune(prog[:off[1]], off[:2], str(path)) == 2
    vals, status, _ = ev.score_batch(prog, off, 0)
    for k in range(len(trees)):
        assert (status[k::len(trees)] == st1[k]).all(), k
        assert (vals[k::len(trees)].view(np.uint64) == alone.view(np.uint64)[k]).all(), k
    ev.close()
