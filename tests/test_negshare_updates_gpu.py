"""The shared-negative pair kernel (dg_sgns_negshare.cu) run by one warp, measured against what a run changes.

The rows of test_negshare_pair_gpu.py are mostly their initial values, so here the
difference from the sequential run is taken relative to the update, on walks that
step back (a, b, a, c, a: the two pairs of a turn often hold one word) at a large
learning rate.  Rounding in another order leaves 1e-6 of the update.  A sum that
rounds across a boundary of the sigmoid table changes its gradient by 0.25 / 83 of
alpha, one term of some 1,400 pairs' (0.003 / 0.5 / sqrt(1400) = 1.6e-4 of the
update at most; a NumPy model of the rule shows 2e-6 to 9e-5 in one run of four);
the bound, 2e-4, allows for it.  In that model the rows are 1.7e-3 off where lanes
without columns keep lane 0's gradient (sizes 65, 100, 200), 3.8e-3 where the second
pair of one word misses the first one's update, and 3e-3 where it reads the
negatives from before it."""
import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
V = 60


def _stepping_back(n_walks, length, seed):
    rng = np.random.default_rng(seed)
    walks = []
    for k in range(n_walks):
        w = rng.integers(0, V, size=length)
        if k % 2 == 0:
            w[2::2] = w[0]
        else:
            w[3::4] = w[1::4][:w[3::4].size]
        walks.append(w)
    return (np.arange(n_walks + 1) * length).astype(np.uint64), np.concatenate(walks).astype(np.uint32)


def _of_the_update(rows, want, init):
    return float(np.linalg.norm(rows.astype(np.float64) - want) / np.linalg.norm(want.astype(np.float64) - init))


@pytest.mark.parametrize("negative", [3, 4, 5, 8])
@pytest.mark.parametrize("size", [64, 65, 100, 128, 130, 200, 250, 256])
def test_one_warp_makes_the_sequential_update(distger_lib, size, negative):
    offs, verts = _stepping_back(10, 16, size)
    counts = np.random.default_rng(1).integers(1, 200, size=V).astype(np.uint32)
    rng = np.random.default_rng(2)
    init = [rng.normal(size=(V, size)).astype(np.float32) * np.float32(0.3) for _ in range(2)]
    got = []
    for kw in (dict(deterministic=True), dict(workers=1)):
        s = SGNS(V, counts, size=size, window=5, negative=negative, sample=0, alpha=0.05, min_count=0, seed=5,
                 table_size=100_000, mode="sg_shared", **kw)
        s.set_rows(*init)
        s.train_host(offs, verts)
        got.append((s.embedding()[0], s.output_rows()))
        s.close()
    for k in range(2):
        assert _of_the_update(got[1][k], got[0][k], init[k]) < 2e-4
