"""The adjoint kernel's loss and gradient against FP64 where its layout changes: every
row size, minibatches of 1 pair, of a few, across the 32 pairs whose ids a warp holds
at once (40, 65) and a last one that is short, the negative count with its own
instance (5) and others (0, 3, 16), runs of one output row and none.  Bounds as in
test_adjoint_gpu.py: loss within 1e-6 relative, gradients within 1e-5 (Frobenius)."""
import numpy as np
import pytest

from distger.sgns import SGNS

pytestmark = pytest.mark.gpu
V = 300


SHAPES = [(32, 1, 5, 7), (64, 21, 5, 300), (128, 40, 5, 333), (128, 65, 3, 200), (256, 33, 0, 100), (256, 5, 16, 64)]


@pytest.mark.parametrize("mode,size,batch,negative,n_pairs", [(m, *s) for m in ("plain", "minibatch") for s in SHAPES] +
                         [("plain", 512, 21, 5, 50)])
def test_loss_and_gradient(distger_lib, oracle, mode, size, batch, negative, n_pairs):
    rng = np.random.default_rng(size + batch)
    counts = rng.integers(1, 50, size=V).astype(np.uint32)
    s = SGNS(V, counts, size=size, window=5, negative=min(negative, 14), sample=0, alpha=0.01, min_count=0, mode=mode,
             seed=3, table_size=10_000, master_rows=40 if mode == "minibatch" else 0)
    scale = 0.7 / np.sqrt(size)
    s.set_rows(rng.normal(size=(V, size)).astype(np.float32) * scale, rng.normal(size=(V, size)).astype(np.float32) * scale)
    inp = rng.integers(0, V, size=n_pairs).astype(np.uint32)
    out = np.repeat(rng.integers(0, V, size=n_pairs), rng.integers(1, 9, size=n_pairs))[:n_pairs].astype(np.uint32)
    neg = rng.integers(0, V, size=(n_pairs + batch - 1) // batch * negative).astype(np.uint32)
    loss, gi, go = s.loss_grad(inp, out, neg, batch=batch, negative=negative)
    v, u = s.embedding()[0].astype(np.float64), s.output_rows().astype(np.float64)
    loss64, gi64, go64 = oracle.sgns_loss_grad(v, u, inp, out, neg, batch, negative)
    assert loss == pytest.approx(loss64, rel=1e-6)
    for g, g64 in ((gi, gi64), (go, go64)):
        assert np.linalg.norm(g - g64) / np.linalg.norm(g64) < 1e-5
    again = s.loss_grad(inp, out, neg, batch=batch, negative=negative)
    assert again[0] == loss and np.array_equal(again[1], gi) and np.array_equal(again[2], go)
