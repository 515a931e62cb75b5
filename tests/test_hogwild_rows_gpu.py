"""Hogwild rows of the kernel that a call takes, against those of the kernels that train one pair
(centre) at a time.

A Hogwild run depends on which updates see each other, so a kernel that trains faster
also trains a little differently.  Measured here: how far the rows of the kernel that a
call takes end from those of the one-at-a-time kernel, over how far two equal runs of
that kernel end from each other (the median of six pairs of runs).  Where the call takes
the one-at-a-time kernel itself this is 1 but for chance (medians of 0.9 to 1.1): at most
1.5.  Where it takes the shared-negative pair kernel, at most 4.

The one-at-a-time kernel is reached with the same tokens: one more walk, longer than the
pair kernel takes, of a vertex that is not in the vocabulary.  Rows and learning rate are
those of a job's last rounds."""
import itertools

import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
V = 22_000


@pytest.fixture(scope="module")
def corpus(distger_lib):
    from distger import WalkEngine, graphgen
    edges = graphgen.chung_lu(V, 110_000, 2.2, seed=9)
    eng = WalkEngine(seed=3)
    eng.load_graph(V, "", make_undirected=True, edges=edges)
    counts = np.add(*eng.graph.degrees())
    paths = eng.run_round(V, 2)
    offs, verts = paths.to_numpy()
    paths.close()
    return np.append(counts, 0).astype(np.uint32), offs, verts


def _rows(corpus, one_at_a_time, **kw):
    counts, offs, verts = corpus
    extra = 70 if one_at_a_time else 2
    s = SGNS(V + 1, counts, sample=1e-3, alpha=0.01, min_count=1, seed=5, table_size=1_000_000, **kw)
    rng = np.random.default_rng(1)
    s.set_rows(*(rng.normal(size=(s.vocab_size, s.size)).astype(np.float32) * np.float32(0.1) for _ in range(2)))
    s.train_host(np.append(offs, offs[-1] + extra), np.append(verts, np.full(extra, V, np.uint32)), 0.0015)
    got = s.embedding()[0].astype(np.float64), s.output_rows().astype(np.float64)
    s.close()
    return got


def _ratios(corpus, **kw):
    one = [_rows(corpus, True, **kw) for _ in range(4)]
    own = [_rows(corpus, False, **kw) for _ in range(3)]
    for k in range(2):
        among = np.median([np.linalg.norm(a[k] - b[k]) for a, b in itertools.combinations(one, 2)])
        yield float(np.median([np.linalg.norm(a[k] - b[k]) for a, b in itertools.product(own, one)]) / among)


@pytest.mark.parametrize("size,window,negative,most", [
    (64, 8, 3, 1.5), (100, 9, 3, 1.5), (128, 5, 5, 1.5), (200, 10, 5, 4), (256, 6, 4, 4), (200, 8, 3, 1.5), (64, 7, 7, 1.5),
    (64, 9, 8, 1.5), (256, 5, 7, 1.5), (128, 5, 2, 1.5)])
def test_shared_negatives(corpus, size, window, negative, most):
    assert max(_ratios(corpus, mode="sg_shared", size=size, window=window, negative=negative)) <= most


@pytest.mark.parametrize("size,window,negative,hs", [
    (32, 6, 5, False), (64, 10, 5, False), (100, 8, 5, False), (128, 5, 1, False), (128, 9, 5, True), (64, 8, 8, True),
    (256, 7, 3, True), (200, 9, 5, False), (256, 5, 5, False), (64, 9, 8, False), (128, 10, 7, False)])
def test_cbow(corpus, size, window, negative, hs):
    assert max(_ratios(corpus, mode="cbow", size=size, window=window, negative=negative, hs=hs)) <= 1.5
