"""Rows that hold infinities: the kernels that train two centres or pairs at a time, run by one
warp, against the one-at-a-time kernels, which one walk more of a vertex outside the
vocabulary brings in (test_hogwild_rows_gpu.py).  Where a value is infinite or no number
afterwards is the same, and the others agree as in test_cbow_updates_gpu.py: the scores
of an infinite column are infinite, so what follows from it has no rounding."""
import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
V = 40


def _run(extra, init, walks, **kw):
    offs = np.arange(len(walks) + 1) * walks.shape[1]
    s = SGNS(V + 1, np.append(np.random.default_rng(1).integers(1, 200, size=V), 0).astype(np.uint32), window=kw.pop("window"),
             sample=0, alpha=0.01, min_count=1, seed=5, table_size=100_000, workers=1, **kw)
    s.set_rows(*(x[:s.vocab_size] for x in init))
    s.train_host(np.append(offs, offs[-1] + extra).astype(np.uint64),
                 np.append(walks.ravel(), np.full(extra, V)).astype(np.uint32))
    got = s.embedding()[0], s.output_rows()
    s.close()
    return got


@pytest.mark.parametrize("mode,size,window,negative,hs", [
    ("cbow", 128, 5, 5, False), ("cbow", 100, 5, 3, False), ("cbow", 64, 1, 5, False), ("cbow", 128, 4, 5, True),
    ("cbow", 200, 4, 3, True), ("sg_shared", 128, 4, 5, False), ("sg_shared", 100, 5, 4, False), ("sg_shared", 200, 3, 3, False)])
@pytest.mark.parametrize("where", ["input", "output"])
def test_infinities_stay_where_they_are(distger_lib, mode, size, window, negative, hs, where):
    rng = np.random.default_rng(size + window)
    walks = rng.integers(0, V, size=(3, 7))
    walks[1, 2::2] = walks[1, 0]
    walks[2, -2:] = 0, 1   # the most frequent words' rows (ids are by count)
    init = [rng.normal(size=(V + 1, size)).astype(np.float32) * np.float32(0.1) for _ in range(2)]
    table = init[0 if where == "input" else 1]
    table[[3, 11, 25], 2] = np.inf, -np.inf, np.inf
    table[7, size - 1] = np.inf
    two = _run(2, init, walks, mode=mode, size=size, window=window, negative=negative, hs=hs)
    one = _run(70, init, walks, mode=mode, size=size, window=window, negative=negative, hs=hs)
    for a, b in zip(two, one):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        np.testing.assert_array_equal(np.isposinf(a), np.isposinf(b))
        np.testing.assert_array_equal(np.isneginf(a), np.isneginf(b))
        fine = np.isfinite(b)
        np.testing.assert_allclose(a[fine], b[fine], atol=2e-5, rtol=0)
