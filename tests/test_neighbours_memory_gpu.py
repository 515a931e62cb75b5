"""Common neighbours where device memory is short: a call fits where 88 bytes an edge do (what
an array for each step, freed in turn, comes to), and where only the bitmaps of the longest
rows do not fit it answers without them.  And rows of two lengths of which only the longer
ones get a bitmap.  Counts equal to those of an empty GPU, and to the CPU restatement of
the reference's gcn tool."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(v, n, seed):
    rng = np.random.default_rng(seed)
    return ((rng.random(n) ** 3 * v).astype(np.uint32), rng.integers(0, v, size=n).astype(np.uint32))


# Bytes left free: 88 an edge and 16 MB for the driver; what the bitmaps leave no room for.
@pytest.mark.parametrize("undirected,left", [(True, 88 * 4_000_000 + (16 << 20)), (True, 66 * 4_000_000 + (24 << 20)),
                                             (False, 66 * 4_000_000 + (16 << 20))])
def test_little_memory(distger_lib, undirected, left):
    import torch
    from distger.synth import common_neighbours
    s, d = _edges(400_000, 4_000_000, 3)
    want = common_neighbours(s, d, 400_000, undirected=undirected)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        got = common_neighbours(s, d, 400_000, undirected=undirected)
    finally:
        del held
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got, want)


def test_only_the_longer_rows_fit(distger_lib, oracle):
    """20 million vertices: 26 bitmaps fit.  10 rows of about 600 entries get one, 40 of about 300 none."""
    from distger.synth import common_neighbours
    v = 20_000_000
    rng = np.random.default_rng(8)
    ids = rng.choice(v, size=3000, replace=False)
    src = np.concatenate([np.repeat(ids[:10], 600), np.repeat(ids[10:50], 300), ids[rng.integers(0, 3000, size=400)], ids[:50]])
    dst = np.concatenate([rng.choice(ids, size=src.size - 50), ids[:50]])
    order = rng.permutation(src.size)
    s, d = src[order].astype(np.uint32), dst[order].astype(np.uint32)
    want = oracle.common_neighbours(s, d, v, undirected=True)
    assert want.max() > 0
    np.testing.assert_array_equal(common_neighbours(s, d, v), want)
