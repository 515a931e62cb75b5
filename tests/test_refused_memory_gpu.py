"""Calls that are refused for want of device memory and made again: the GPU is filled, the call
ends with DG_ERR_NOMEM, the memory is given back, and the same handle answers as one that
was never refused (its kept buffers are asked for again).  Sizes are such that the refused
allocation cannot come from a page that the driver already holds."""
import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
NOMEM = -4


@pytest.fixture
def full():
    """A call while the GPU is full: its error's code, None if it succeeded."""
    import torch

    def call(f):
        from distger._lib import DistgerError
        torch.cuda.synchronize()
        held, piece = [], 64 << 30
        while piece >= 1 << 20:
            try:
                held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                piece //= 2
        try:
            f()
        except DistgerError as e:
            return e.code
        finally:
            del held
            torch.cuda.empty_cache()
        return None
    return call


def _trainer(v, **kw):
    s = SGNS(v, np.full(v, 10, np.uint32), size=128, window=5, negative=5, sample=0, alpha=0.01, min_count=0, seed=3,
             table_size=10_000, **kw)
    rng = np.random.default_rng(v)
    s.set_rows(*(rng.normal(size=(v, 128)).astype(np.float32) * np.float32(0.1) for _ in range(2)))
    return s


def test_rows_of_the_bf16_form(distger_lib, full):
    s, other = _trainer(80_000, mode="plain_bf16"), _trainer(80_000, mode="plain_bf16")
    want = other.embedding()[0]
    assert full(s.embedding) == NOMEM
    np.testing.assert_array_equal(s.embedding()[0], want)
    np.testing.assert_array_equal(s.output_rows(), other.output_rows())


def test_gradient(distger_lib, full):
    rng = np.random.default_rng(1)
    n = 2_100_000
    ids = [rng.integers(0, 80_000, size=k).astype(np.uint32) for k in (n, n, n // 21 * 5)]
    few = [ids[0][:2100], ids[1][:2100], ids[2][:500]]
    s, other = _trainer(80_000, mode="plain"), _trainer(80_000, mode="plain")
    s.loss_grad(*few, batch=21, negative=5)   # buffers for the small call
    assert full(lambda: s.loss_grad(*ids, batch=21, negative=5)) == NOMEM
    for k, x in enumerate(other.loss_grad(*ids, batch=21, negative=5)):
        np.testing.assert_array_equal(s.loss_grad(*ids, batch=21, negative=5)[k], x)


def test_walks_of_another_length(distger_lib, oracle, full):
    from distger import WalkEngine, graphgen
    edges = graphgen.chung_lu(300, 900, 2.1, seed=4)
    eng = WalkEngine(seed=7, max_len=64)
    eng.load_graph(300, "", make_undirected=True, edges=edges)
    eng.run_round(300, 1).close()
    eng.max_len = 6000
    assert full(lambda: eng.run_round(300, 2)) == NOMEM
    want, _ = oracle.walk_rounds(oracle.Csr(edges, 300, undirected=True), 300, 20, 5, 3, seed=7)
    for r, max_len in ((2, 64), (3, 6000)):
        eng.max_len = max_len
        paths = eng.run_round(300, r)
        offs, verts = paths.to_numpy()
        paths.close()
        np.testing.assert_array_equal(offs, want[r - 1][0])
        np.testing.assert_array_equal(verts, want[r - 1][1])
