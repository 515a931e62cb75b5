"""What a user of this framework has it do, as cases that can be timed and compared.

The job of the framework is a node embedding: walk rounds over a graph streamed
into a skip-gram or CBOW trainer, on graphs from ten thousand to a million
vertices, with word2vec's or dsgl's flags.  The cases are that job's rounds under
each training rule, the walks alone, the loss gradient, and the edge-data
precompute.  Graphs are power laws of the shapes in distger.graphgen.CONFIGS,
generated on the GPU from the seed; trainers hold rows of the scale that they
have late in a job, and its learning rate there.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gdistger-re_b200"))

import distger  # noqa: E402
from distger import _lib  # noqa: E402
from distger.adjoint import pairs_from_walks  # noqa: E402
from distger.sgns import SGNS  # noqa: E402
from distger.synth import common_neighbours  # noqa: E402
from distger.walk import EDGE_DTYPE  # noqa: E402

# Vertices, edge draws, power-law exponent and degree cap of the graphs of
# distger.graphgen.CONFIGS that the cases use.
SMALL = dict(v=10_000, m=100_000, beta=2.2, cap=0)
MIDDLE = dict(v=50_000, m=500_000, beta=2.2, cap=0)
YOUTUBE = dict(v=1_138_499, m=2_990_443, beta=2.1, cap=28_000)
LIVEJOURNAL = dict(v=2_238_731, m=14_000_000, beta=2.3, cap=0)

TOKENS_PER_WALK = 22   # footprints: the entropy test ends nearly every walk at the first step it may
SCALE = 0.1            # rms of a row's elements late in a job
ALPHA = 0.0015         # learning rate of a job's last rounds: 0.025 exp(-0.1 round) at the 28th


def listed():
    return [
        # The smallest call: one round of walks over a small graph, brought to the host.
        dict(SMALL, name="walk_small", kind="walk", walkers=10_000),
        # A corpus of walks of a YouTube-sized graph for another program (the walk file's content).
        dict(YOUTUBE, name="walk_youtube", kind="walk", walkers=1_138_499),
        # Walk rounds whose visit counts and entropies are what is wanted (how many rounds does a graph need).
        dict(LIVEJOURNAL, name="visits_livejournal", kind="visits", rounds=2),
        # The reference job's default rule (-cbow 1) with the flags of its run.sh (-size 100) on a small graph.
        dict(SMALL, name="cbow_small", kind="train", mode="cbow", size=100, window=10, negative=5, rounds=3),
        # The same rule at the size of the paper's graphs: word2vec.cu's default trainer.
        dict(YOUTUBE, name="cbow_youtube", kind="train", mode="cbow", size=128, window=10, negative=5, rounds=2),
        # Skip-gram with per-pair negatives on FP32 rows (-cbow 0 -reuse-neg 0).
        dict(YOUTUBE, name="plain_youtube", kind="train", mode="plain", size=128, window=10, negative=5, rounds=1),
        # The same on BF16 rows, the benchmark's form.
        dict(YOUTUBE, name="plain_bf16_youtube", kind="train", mode="plain_bf16", size=128, window=10, negative=5,
             rounds=1),
        # dsgl's minibatch rule, DistGER's own trainer.
        dict(YOUTUBE, name="minibatch_youtube", kind="train", mode="minibatch", size=128, window=10, negative=5,
             rounds=1),
        # Skip-gram with one negative set per walk (-cbow 0 -reuse-neg 1), word2vec.cu's other size, its default window.
        dict(MIDDLE, name="shared_middle", kind="train", mode="sg_shared", size=200, window=5, negative=5, rounds=1),
        # Hierarchical softmax beside the negatives (-hs 1) on the default rule.
        dict(MIDDLE, name="cbow_hs_middle", kind="train", mode="cbow", size=128, window=5, negative=5, rounds=1, hs=True),
        # Loss and gradient of explicit minibatches (a user's own optimiser on top of it).
        dict(MIDDLE, name="gradient_middle", kind="gradient", mode="plain", size=128, window=10, negative=5,
             pairs=200_000),
        # The edge data of the walk: common-neighbour counts of every edge, host to host.
        dict(YOUTUBE, name="neighbours_youtube", kind="neighbours"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    v = _log_int(rng, 10_000, 1_100_000)
    c = dict(v=v, m=int(v * rng.uniform(2.6, 10.0 if v < 300_000 else 3.0)), beta=round(rng.uniform(2.1, 2.3), 3),
             cap=28_000)
    kind = rng.choice(["walk", "visits", "train", "train", "train", "train", "train", "train", "gradient", "neighbours"])
    c["kind"] = kind
    if kind == "walk":
        c["walkers"] = _log_int(rng, min(v, 10_000), v)
    elif kind == "visits":
        c["rounds"] = rng.randint(1, 3)
    elif kind == "train":
        mode = rng.choice(["cbow", "cbow", "plain", "plain_bf16", "minibatch", "sg_shared"])
        c.update(mode=mode, window=rng.randint(5, 10), negative=rng.choice([3, 5, 5, 7, 8]), rounds=1)
        c["size"] = rng.choice([64, 128, 128, 256] if mode in ("plain_bf16", "minibatch") else [64, 100, 128, 200])
        c["v"] = min(v, {"cbow": 1_100_000, "sg_shared": 200_000, "minibatch": 300_000}.get(mode, 500_000))
        if mode == "cbow" and rng.random() < 0.25:
            c["hs"] = True
        c["m"] = int(c["v"] * rng.uniform(2.6, 10.0 if c["v"] < 300_000 else 3.0))
    elif kind == "gradient":
        c.update(v=min(v, 200_000), mode=rng.choice(["plain", "minibatch"]), size=rng.choice([64, 128, 256]), window=10,
                 negative=rng.choice([3, 5, 5, 8]), pairs=_log_int(rng, 20_000, 400_000))
        c["m"] = int(c["v"] * rng.uniform(2.6, 10.0))
    return c


def _edges(case, seed, count=0):
    """Undirected power-law edge list without loops, host records: each pair once and no isolated vertex, or,
    with a count, that many records as they come (where the graph has too few, the first ones again)."""
    g = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 17)
    v, m = case["v"], case["m"]
    w = (np.arange(v, dtype=np.float64) + 1.0) ** (-1.0 / (case["beta"] - 1.0))
    w *= 2.0 * m / w.sum()
    if case["cap"]:
        np.minimum(w, case["cap"], out=w)
    cdf = np.cumsum(w)   # on the host, where a sum's order is always the same
    cdf = torch.from_numpy(cdf / cdf[-1]).cuda()

    def ends(n):
        u = torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
        return torch.searchsorted(cdf, u, right=True).clamp_(max=v - 1)

    s, d = ends(m + count // 4), ends(m + count // 4)
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    key = torch.unique((lo * v + hi)[lo != hi])
    if count:
        key = key[torch.randperm(key.numel(), device="cuda", generator=g)]
        key = torch.cat([key, key])[:count]
    s, d = key // v, key % v
    deg = torch.bincount(s, minlength=v) + torch.bincount(d, minlength=v)
    alone = torch.nonzero(deg == 0).flatten()[:0 if count else v]
    mate = ends(alone.numel())
    mate = torch.where(mate == alone, (mate + 1) % v, mate)
    s, d = torch.cat([s, alone]), torch.cat([d, mate])
    name = torch.randperm(v, device="cuda", generator=g)
    order = torch.randperm(s.numel(), device="cuda", generator=g)
    rec = torch.empty((s.numel(), 3), dtype=torch.int32, device="cuda")
    rec[:, 0] = name[s[order]].int()
    rec[:, 1] = name[d[order]].int()
    rec[:, 2] = (1.0 - torch.rand(s.numel(), device="cuda", generator=g)).view(torch.int32)
    return rec.cpu().numpy().reshape(-1).view(EDGE_DTYPE)


def _rows(n, size, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(n, size, device="cuda", generator=g) * SCALE).cpu().numpy()


def _engine(case, seed):
    eng = distger.WalkEngine(seed=seed)
    eng.load_graph(case["v"], "", make_undirected=True, edges=_edges(case, seed))
    return eng


def _trainer(case, seed, counts):
    return SGNS(case["v"], counts, size=case["size"], window=case["window"], negative=case["negative"], batch_size=21,
                sample=1e-3, alpha=0.01, min_count=0, mode=case["mode"], seed=seed, hs=case.get("hs", False))


def _pinned(*shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "round": 2}
    if kind == "neighbours":
        e = _edges(case, seed, case["m"])
        st.update(src=np.ascontiguousarray(e["src"]), dst=np.ascontiguousarray(e["dst"]))
        return st
    eng = _engine(case, seed)
    st["engine"] = eng
    if kind == "walk":
        st["offsets"] = _pinned(case["walkers"] + 1, dtype=torch.int64)
        st["vertices"] = _pinned(case["walkers"] * eng.max_len, dtype=torch.int32)
    elif kind == "train":
        s = _trainer(case, seed, np.add(*eng.graph.degrees()))
        s.set_rows(_rows(s.vocab_size, s.size, 2 * seed), _rows(s.vocab_size, s.size, 2 * seed + 1))
        st.update(sgns=s, input=_pinned(s.vocab_size, s.size), output=_pinned(s.vocab_size, s.size))
    elif kind == "gradient":
        s = _trainer(case, seed, np.add(*eng.graph.degrees()))
        vi, vo = _rows(s.vocab_size, s.size, 2 * seed), _rows(s.vocab_size, s.size, 2 * seed + 1)
        s.set_rows(vi, vo)
        walks = eng.run_round(case["v"], 2, n_walkers=min(case["v"], case["pairs"] // 100 + 100))
        t = s.tables()
        inp, out, neg = pairs_from_walks(*walks.to_numpy(), t["v2w"], t["table"], window=case["window"], batch=21,
                                         negative=case["negative"], n_pairs=case["pairs"], seed=seed)
        walks.close()
        st.update(sgns=s, pairs=SGNS._pairs(inp, out, neg, 21, case["negative"]),
                  grad_in=_pinned(s.vocab_size, s.size), grad_out=_pinned(s.vocab_size, s.size))
    return st


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "neighbours":
        return common_neighbours(st["src"], st["dst"], case["v"])
    eng = st["engine"]
    if kind == "walk":
        paths = eng.run_round(case["walkers"], st["round"])
        st["round"] += 1
        off, ver = st["offsets"], st["vertices"]
        _lib.check(distger.lib().dg_paths_copy(paths.handle, off.data_ptr(), ver.data_ptr()))
        n = paths.info.footprints
        paths.close()
        return {"offsets": off, "vertices": ver[:n]}
    if kind == "visits":
        done = []
        for _ in range(case["rounds"]):
            paths = eng.run_round(case["v"], st["round"])
            st["round"] += 1
            i = paths.info
            done += [i.steps, i.draws, i.traces, i.relative_entropy]
            paths.close()
        return {"rounds": done, "visits": eng.graph.visits()}
    if kind == "train":
        s = st["sgns"]
        for _ in range(case["rounds"]):
            paths = eng.run_round(case["v"], st["round"])
            st["round"] += 1
            s.train_paths(paths, ALPHA)
            paths.close()
        _lib.check(distger.lib().dg_sgns_copy_embedding(s.handle, st["input"].data_ptr(), None, None))
        _lib.check(distger.lib().dg_sgns_copy_output(s.handle, st["output"].data_ptr()))
        return {"input": st["input"], "output": st["output"]}
    loss = C.c_double()
    _lib.check(distger.lib().dg_sgns_loss_grad(st["sgns"].handle, C.byref(st["pairs"][0]), C.byref(loss),
                                               st["grad_in"].data_ptr(), st["grad_out"].data_ptr()))
    return {"loss": loss.value, "input": st["grad_in"], "output": st["grad_out"]}


def _pairs_per_token(case):
    """Mean number of contexts of a centre: both sides of a shrunk window in a walk of TOKENS_PER_WALK."""
    n, w = TOKENS_PER_WALK, case["window"]
    spans = [w] if case["mode"] == "sg_shared" else range(1, w + 1)
    return sum(min(p, s) + min(n - 1 - p, s) for s in spans for p in range(n)) / (n * len(spans))


def work(case):
    kind, v, m = case["kind"], case["v"], 2 * case["m"]
    csr = 8.0 * v + 8.0 * m   # row bounds, then a neighbour and its edge data
    if kind == "neighbours":
        return {"bytes": 12.0 * case["m"], "flops": 0.0}
    if kind == "walk":
        return {"bytes": csr + 4.0 * TOKENS_PER_WALK * case["walkers"], "flops": 0.0}
    if kind == "visits":
        return {"bytes": case["rounds"] * (csr + 8.0 * v), "flops": 0.0}
    d, n = case["size"], case["negative"]
    if kind == "gradient":
        return {"bytes": 4.0 * d * v * 4 + 8.0 * case["pairs"], "flops": 6.0 * d * (1 + n) * case["pairs"]}
    tokens = float(TOKENS_PER_WALK) * v
    each = 2.0 if case["mode"] in ("plain_bf16", "minibatch") else 4.0
    per_round = csr + 4.0 * tokens + 4.0 * each * d * v   # both tables read and written
    if case["mode"] == "cbow":
        flops = tokens * d * (6.0 * (1 + n) + 2.0 * _pairs_per_token(case))
    else:
        flops = tokens * _pairs_per_token(case) * 6.0 * d * (1 + n)
    return {"bytes": case["rounds"] * per_round + 8.0 * d * v, "flops": case["rounds"] * flops}


def exact(case, seed):
    """The gradient in 64 bits.  Training by racing workers and the walks' whole numbers have no such value."""
    if case["kind"] != "gradient":
        return None
    st = prepare(case, seed)
    s, (inp, out, neg) = st["sgns"], st["pairs"][1]
    v, u = (torch.from_numpy(_rows(s.vocab_size, s.size, 2 * seed + k)).cuda() for k in (0, 1))
    if case["mode"] == "minibatch":   # BF16 rows beyond the 65,536 most frequent words
        for t in (v, u):
            t[65536:] = t[65536:].bfloat16().float()
    v, u = v.double(), u.double()
    i, o = (torch.from_numpy(x.astype(np.int64)).cuda() for x in (inp, out))
    k = torch.from_numpy(neg.astype(np.int64)).cuda().view(-1, case["negative"])
    gi, go = torch.zeros_like(v), torch.zeros_like(u)
    loss = 0.0
    for a in range(0, i.numel(), 21 * 1000):   # whole minibatches at a time
        b = min(a + 21 * 1000, i.numel())
        nk = k[torch.arange(a, b, device="cuda") // 21]
        x = v[i[a:b]]
        pos, vn = u[o[a:b]], u[nk]
        sp, sn = (x * pos).sum(1), torch.einsum("pd,pkd->pk", x, vn)
        loss += float(torch.nn.functional.softplus(-sp).sum() + torch.nn.functional.softplus(sn).sum())
        gp, gn = torch.sigmoid(sp) - 1.0, torch.sigmoid(sn)
        gi.index_add_(0, i[a:b], gp[:, None] * pos + torch.einsum("pk,pkd->pd", gn, vn))
        go.index_add_(0, o[a:b], gp[:, None] * x)
        go.index_add_(0, nk.flatten(), (gn[:, :, None] * x[:, None, :]).flatten(0, 1))
    return {"loss": loss, "input": gi, "output": go}
