"""The walk kernel's tabulated step terms and footprint cache, at the lengths where
they change: walks bit-exact against the CPU checker (whose state is divided and
carried step by step) for termination tests from the first step on (min_len 1) and
long after the cached footprints end (min_len 60), with every launch shape (16 to 48
cached footprints), on a graph of many step-backs and on one of hubs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", range(6))
@pytest.mark.parametrize("min_len,max_len", [(1, 64), (16, 64), (25, 64), (60, 200)])
def test_walks_bit_exact(distger_lib, oracle, min_len, max_len, shape):
    from distger import WalkEngine, graphgen
    from distger._lib import check, lib
    for n, m, beta in ((300, 900, 2.1), (400, 6000, 2.4)):
        edges = graphgen.chung_lu(n, m, beta, seed=min_len)
        eng = WalkEngine(seed=77, max_len=max_len)
        eng.set_minLength(min_len)
        eng.set_init_round(2)
        eng.load_graph(n, "", make_undirected=True, edges=edges)
        check(lib().dg_walk_set_shape(eng.graph.handle, shape))
        want, _ = oracle.walk_rounds(oracle.Csr(edges, n, undirected=True), n, min_len, 2, 2, seed=77)
        for r in (1, 2):
            paths = eng.run_round(n, r)
            offs, verts = paths.to_numpy()
            paths.close()
            np.testing.assert_array_equal(offs, want[r - 1][0])
            np.testing.assert_array_equal(verts, want[r - 1][1])
