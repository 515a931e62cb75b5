"""The Hogwild shared-negative kernel that trains two pairs at a time (dg_sgns_negshare.cu), one warp.

One warp sees every update of its own, so its run is the sequential one
(deterministic = 1, sgns_negshare_kernel, itself bit-exact against the CPU
restatement) but for the order of its sums.  Rows may differ by what that
rounding can do: the bound is the 2e-3 relative Frobenius norm that FP32 rows
keep against FP64 ones (a sum that rounds across a boundary of the 83-per-unit
sigmoid table takes its neighbour).  Walks of 0, 1, 2, 63 and 64 tokens, words
that repeat within a window and within a walk's negatives (a table of few
words), every row size, padded sizes, and each end of the window and negative
ranges.
"""
import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
V = 60


def _walks(max_len, seed):
    rng = np.random.default_rng(seed)
    lens = np.concatenate([[0, 1, 2, max_len - 1, max_len], rng.integers(2, max_len + 1, size=40)])
    walks = [rng.integers(0, V, size=n) for n in lens]
    for w in walks[5::3]:   # a word stepped back to, as a walk does
        w[2::2] = w[0]
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64), np.concatenate(walks).astype(np.uint32)


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64)))


CASES = [(64, 1, 1, 32), (64, 5, 5, 64), (100, 10, 5, 22), (128, 10, 0, 40), (128, 64, 8, 64), (200, 5, 5, 22),
         (200, 7, 8, 22), (256, 3, 5, 5), (256, 2, 3, 63), (128, 10, 5, 65), (128, 10, 9, 32), (32, 4, 5, 20)]


@pytest.mark.parametrize("size,window,negative,max_len", CASES)
def test_one_warp_is_the_sequential_run(distger_lib, size, window, negative, max_len):
    offs, verts = _walks(max_len, size + window)
    counts = np.random.default_rng(1).integers(1, 200, size=V).astype(np.uint32)
    rng = np.random.default_rng(2)
    init = [rng.normal(size=(V, size)).astype(np.float32) * 0.3 for _ in range(2)]
    out = []
    for kw in (dict(deterministic=True), dict(workers=1)):
        s = SGNS(V, counts, size=size, window=window, negative=negative, sample=0, alpha=0.01, min_count=0, seed=5,
                 table_size=100_000, mode="sg_shared", **kw)
        s.set_rows(*init)
        info = s.train_host(offs, verts)
        out.append((s.embedding()[0], s.output_rows(), (info.words, info.trained, info.pairs)))
        s.close()
    (i0, o0, n0), (i1, o1, n1) = out
    assert n0 == n1
    assert _rel(i1, i0) < 2e-3 and _rel(o1, o0) < 2e-3
