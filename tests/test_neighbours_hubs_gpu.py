"""Common-neighbour counts where the look-up of the longer row changes: rows below and
above the 128 entries from which a bitmap may serve, more long rows than the bitmaps'
space holds (a vertex range so wide that 25 fit), repeated edges and self-loops, and
vertex counts at the edges of the sort keys' bits, against the CPU restatement of the
reference's gcn tool.  Whole numbers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(v, hubs, degree, seed, repeat=0):
    rng = np.random.default_rng(seed)
    ids = rng.choice(v, size=min(v, 3000), replace=False)
    h = ids[:hubs]
    src = np.repeat(h, degree)
    dst = rng.choice(ids, size=src.size)
    extra = rng.choice(ids, size=(2, 400))
    s, d = np.concatenate([src, extra[0]]), np.concatenate([dst, extra[1]])
    if repeat:
        s, d = np.concatenate([s, d[:repeat], s[:3]]), np.concatenate([d, s[:repeat], s[:3]])   # mirrored, loops
    order = rng.permutation(s.size)
    return s[order].astype(np.uint32), d[order].astype(np.uint32)


@pytest.mark.parametrize("v,hubs,degree,repeat", [(65, 3, 40, 20), (64, 4, 200, 50), (4096, 6, 127, 0), (4097, 6, 128, 30),
                                                   (5000, 30, 700, 100), (20_000_000, 40, 300, 40)])
def test_counts_equal_the_restatement(distger_lib, oracle, v, hubs, degree, repeat):
    from distger.synth import common_neighbours
    s, d = _graph(v, hubs, degree, seed=v % 1000 + hubs, repeat=repeat)
    want = oracle.common_neighbours(s, d, v, undirected=True)
    assert want.max() > 0
    np.testing.assert_array_equal(common_neighbours(s, d, v), want)
