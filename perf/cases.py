"""What this framework's speed is measured on.

Each case is a plain dict: what a user's program has in hand (a graph of a family and size, a pattern, the
residency), and the public call it makes.  `listed` names the fixed cases, `draw` gives others of the same
ranges.  Graphs are the generators' stand-ins for converted datasets, the same families and parameters as
the benchmark's workloads and the test fixtures (Chung-Lu power law, R-MAT .57/.19/.19), with other seeds
for other inputs.

Cases by what they do:
  match     one query through Context.match, counts per pattern (and per root edge where asked)
  replay    a prepared query replayed (Context.prepare, Query.run)
  features  the learned scheduler's root features (root filter included)
  place     a graph placed from host arrays and its root edges listed
  predict   the cost model's predictions for a list of roots
  gradient  the cost model's loss and gradient on a batch
"""
import math

import numpy as np
import torch

import pumatch_b200 as pm
from pumatch_b200 import learn
from pumatch_b200 import patterns as P

SHAPES = {"K4": P.clique(4), "K5": P.clique(5), "C4": P.cycle(4), "C5": P.cycle(5), "C6": P.cycle(6), "S4": P.star(4),
          "P4": P.path(4), "P5": P.path(5), "house": P.house(), "house_tail": P.house_tail(1),
          "C4_tail": P.cycle_tail(4, 1), "C5_tail2": P.cycle_tail(5, 2)}


def listed():
    return [
        # The smallest call: a 4-clique on a graph of a few hundred vertices, where launches and the root
        # filter count, not the search.
        dict(name="clique4_400", do="match", family="chung_lu", vertices=400, edges=2_000, pattern="K4"),
        # An ordinary unlabeled query on a small graph.
        dict(name="house_3000", do="match", family="chung_lu", vertices=3_000, edges=20_000, pattern="house"),
        # Cliques on a skewed graph: many short intersections.
        dict(name="clique5_rmat32k", do="match", family="rmat", vertices=32_768, edges=524_288, pattern="K5"),
        # The benchmark's query family (long cycles, unlabeled) as one shard of a sharded run, with the
        # per-root counts a cost log or a resumable run keeps.
        dict(name="cycle6_20k_shard", do="match", family="chung_lu", vertices=20_000, edges=100_000, pattern="C6",
             shards=64, per_root=True),
        # Cycle plus attachment, unlabeled: fresh sets and copies at the last levels.
        dict(name="housetail_20k_shard", do="match", family="chung_lu", vertices=20_000, edges=100_000,
             pattern="house_tail", shards=64),
        # The reference's default mode, its candidate-set cap included: labeled, truncated at 4,096.
        dict(name="cycle5_lab8_cap4096", do="match", family="rmat", vertices=32_768, edges=524_288, labels=8,
             pattern="C5", pattern_seed=202, truncate=4096),
        # The configured labeled query (5-cycle with a two-vertex tail, 32 labels), in device memory.
        dict(name="cycle5tail_lab32", do="match", family="rmat", vertices=131_072, edges=2_097_152, labels=32,
             pattern="C5_tail2", pattern_seed=202, per_root=True),
        # The same query with the adjacency in host memory: 60% of it in static frames, 28% evictable.
        dict(name="cycle5tail_lab32_paged", do="match", family="rmat", vertices=131_072, edges=2_097_152, labels=32,
             pattern="C5_tail2", pattern_seed=202, pool=0.88, static=0.6, page_kb=16),
        # Twenty patterns of 4 to 7 vertices in one launch, prepared once and replayed.
        dict(name="batch20_lab32_replay", do="replay", family="rmat", vertices=65_536, edges=1_048_576, labels=32,
             pattern="batch20", pattern_seed=303),
        # The learned scheduler's inputs for every root edge of a query.
        dict(name="features_512k", do="features", family="rmat", vertices=524_288, edges=4_194_304, labels=8,
             pattern="C5_tail2", pattern_seed=202),
        # From host arrays to the root list: what a program pays before its first query on a new graph.
        dict(name="place_256k", do="place", family="rmat", vertices=262_144, edges=4_194_304, labels=16,
             pattern="C5", pattern_seed=202),
        # A training step's gradient at the batch size that fitting uses by default.
        dict(name="gradient_8192", do="gradient", samples=8_192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "clique", "long", "labeled", "labeled", "paged", "batch", "features", "place",
                       "predict", "gradient"])
    if kind == "small":  # whole queries on small and middling graphs, unlabeled
        n = _log(rng, 300, 16_000)
        return dict(do=rng.choice(["match", "match", "replay"]), family="chung_lu", vertices=n,
                    edges=int(n * rng.uniform(4.5, 6.0)), pattern=rng.choice(["K4", "K5", "C4", "house", "C4_tail", "P4", "S4"]),
                    per_root=rng.random() < 0.3)
    if kind == "clique":
        n = _log(rng, 4_000, 32_000)
        return dict(do="match", family="rmat", vertices=n, edges=int(n * rng.uniform(8, 15)),
                    pattern=rng.choice(["K4", "K5"]), per_root=rng.random() < 0.3)
    if kind == "long":  # one shard of a long query, unlabeled
        n = _log(rng, 1_500, 20_000)
        return dict(do="match", family="chung_lu", vertices=n, edges=int(n * rng.uniform(4.0, 5.0)),
                    pattern=rng.choice(["C5", "C6", "house_tail", "P5"]), per_root=rng.random() < 0.5,
                    shards=max(1, int((n / 2500) ** 2.2)))
    if kind == "labeled":
        few = rng.random() < 0.3
        n = _log(rng, 4_000, 30_000 if few else 130_000)
        c = dict(do=rng.choice(["match", "match", "replay"]), family="rmat", vertices=n,
                 edges=int(n * rng.uniform(8, 15.5)), labels=rng.randint(8, 12) if few else 32,
                 pattern=rng.choice(["K5", "C5", "house", "P5"] if few else ["K5", "C5", "house", "P5", "C5_tail2"]),
                 pattern_seed=rng.randint(1, 10_000), per_root=rng.random() < 0.3)
        if rng.random() < 0.25:
            c["truncate"] = rng.choice([64, 1024, 4096])
        return c
    if kind == "paged":
        n = _log(rng, 8_000, 130_000)
        static = rng.choice([0.0, 0.3, 0.6])
        return dict(do="match", family="rmat", vertices=n, edges=int(n * rng.uniform(8, 15.5)), labels=32,
                    pattern=rng.choice(["C5", "house", "C5_tail2"]), pattern_seed=rng.randint(1, 10_000),
                    pool=max(static, 0.2) + rng.choice([0.28, 0.5]), static=static, page_kb=rng.choice([16, 64]))
    if kind == "batch":
        n = _log(rng, 4_000, 60_000)
        return dict(do=rng.choice(["match", "replay"]), family="rmat", vertices=n, edges=int(n * rng.uniform(8, 15)),
                    labels=32, pattern="batch20", pattern_seed=rng.randint(1, 10_000))
    if kind in ("features", "place"):
        n = _log(rng, 20_000, 400_000)
        return dict(do=kind, family="rmat", vertices=n, edges=int(n * rng.uniform(5, 8)), labels=rng.randint(6, 32),
                    pattern=rng.choice(["C5", "C5_tail2", "house"]), pattern_seed=rng.randint(1, 10_000))
    return dict(do=kind, samples=_log(rng, 200, 260_000 if kind == "predict" else 40_000))


def _labeled(case):
    return bool(case.get("labels"))


def _host_graph(case, seed):
    n, m = case["vertices"], case["edges"]
    if case["family"] == "chung_lu":
        hg = pm.gen_chung_lu(n, m, seed=seed)
    else:
        hg = pm.gen_rmat(n, m, seed=seed, device=0)
    return pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(n, case["labels"], seed) if _labeled(case) else None)


def _pattern_labels(case):
    return P.seeded_labels(SHAPES[case["pattern"]][0], case["labels"], case["pattern_seed"])


def _patterns(case):
    if case["pattern"] == "batch20":
        texts = [t for _, t in P.batch_of_20(case["pattern_seed"], case["labels"])]
    else:
        k, edges = SHAPES[case["pattern"]]
        texts = [P.to_g(k, edges, _pattern_labels(case) if _labeled(case) else None)]
    return [pm.PatternPreprocessor(text=t, labeled=_labeled(case)) for t in texts]


def _root_cap(case):
    """Room for every root edge any graph of the case can have (how many there are differs by graph)."""
    return 2 * case["edges"] // (case["labels"] // 2 if _labeled(case) else 1)


def _model_data(case, seed):
    """Weights, the features' and targets' scales, inputs and targets of the cost model."""
    g = torch.Generator().manual_seed(seed)
    w = torch.randn(learn.NPARAM, generator=g) * 0.2
    mu, sd = torch.rand(learn.NIN, generator=g) * 4, torch.rand(learn.NIN, generator=g) + 0.5
    x = (torch.randn(case["samples"], learn.NIN, generator=g) * 2 + 3).abs()
    t = torch.randn(case["samples"], learn.NOUT, generator=g)
    return w.numpy(), mu.numpy(), sd.numpy(), x, t


def prepare(case, seed):
    s = {"case": case}
    if case["do"] in ("predict", "gradient"):
        w, mu, sd, x, t = _model_data(case, seed)
        model = learn.CostModel(0, seed=1)
        model.set_weights(w)
        model.mu, model.sd = mu, sd
        model.tmu, model.tsd = np.array([15.0, 6.0], np.float32), np.array([3.0, 2.0], np.float32)
        s.update(model=model, x=x.cuda(), t=t.cuda())
        return s
    hg = _host_graph(case, seed)
    s["patterns"] = _patterns(case)
    s["ctx"] = pm.Context(0)
    if case["do"] == "place":
        s["host"] = hg
        return s
    if case.get("pool"):
        page = case["page_kb"] << 10
        s["graph"] = pm.GraphPreprocessor.from_host(
            hg, labeled=_labeled(case), paged=True, page_bytes=page,
            frame_pool_bytes=max(page, int(hg.colidx.nbytes * case["pool"]) // page * page),
            static_pool_bytes=int(hg.colidx.nbytes * case["static"]) // page * page)
    else:
        s["graph"] = pm.GraphPreprocessor.from_host(hg, labeled=_labeled(case))
    if case["do"] == "features":
        return s
    opts = dict(timeout_ms=60_000)
    if case.get("truncate"):
        opts["truncate"] = case["truncate"]
    if case.get("shards", 1) > 1:
        opts.update(shard_rank=0, shard_count=case["shards"])
    if case.get("per_root"):
        s["per_root"] = torch.zeros(_root_cap(case), dtype=torch.int64, device="cuda")
        opts["root_counts_ptr"] = s["per_root"].data_ptr()
        s["stream"] = torch.cuda.ExternalStream(s["ctx"].stream_ptr)
        torch.cuda.synchronize()
    s["opts"] = opts
    if case["do"] == "replay":
        s["query"] = s["ctx"].prepare(s["graph"], s["patterns"], **opts)
    return s


def run(s):
    do = s["case"]["do"]
    if do == "predict":
        return s["model"].predict(s["x"])
    if do == "gradient":
        loss, grad = s["model"].gradient(s["x"], s["t"])
        return {"loss": loss, "grad": grad}
    if do == "features":
        x = learn.root_features(s["ctx"], s["graph"], s["patterns"][0])
        return torch.nn.functional.pad(x, (0, 0, 0, _root_cap(s["case"]) - x.shape[0]))
    if do == "place":
        g = pm.GraphPreprocessor.from_host(s["host"], labeled=_labeled(s["case"]))
        roots, info = s["ctx"].roots(g, s["patterns"][0]), g.info()
        g.close()
        roots = np.pad(roots, ((0, _root_cap(s["case"]) - len(roots)), (0, 0)))
        return {"roots": roots, "max_degree": info["max_degree"], "n_labels": info["n_labels"]}
    if "per_root" in s:  # the kernel adds to it
        with torch.cuda.stream(s["stream"]):
            s["per_root"].zero_()
    if do == "replay":
        counts, st = s["query"].run()
    else:
        counts, st = s["ctx"].match(s["graph"], s["patterns"], **s["opts"])
    out = {"counts": np.array(counts, dtype=np.uint64).view(np.int64),
           "stats": np.array([st["n_roots"], st["set_ops"], st["alg_bytes"]], dtype=np.uint64).view(np.int64)}
    if "per_root" in s:
        out["per_root"] = s["per_root"]
    return out


def work(case):
    """The graph's arrays read once, the outputs written once; the model's products.  A search's own work
    (its set operations) depends on the graph drawn and is not a number of the case."""
    if "samples" in case:
        n, layers = case["samples"], learn.NIN * 64 + 64 * 64 + 64 * learn.NOUT
        if case["do"] == "predict":
            return {"bytes": 4 * n * (learn.NIN + learn.NOUT) + 2 * learn.NPARAM, "flops": 2 * n * layers}
        return {"bytes": 4 * n * (learn.NIN + learn.NOUT) + 6 * learn.NPARAM,
                "flops": 2 * n * (3 * layers - learn.NIN * 64)}
    nadj, n, labels = 2 * case["edges"], case["vertices"], case.get("labels", 0)
    b = 4 * nadj + 8 * (n + 1) + (n if labels else 0)
    roots = nadj // (labels * labels) if labels else nadj // 2
    if case["do"] == "features":
        b += roots * (8 + 4 * learn.NIN)
    elif case["do"] == "place":
        b += 3 * n + roots * 8  # labels come as 32-bit words
    elif case.get("per_root"):
        b += roots * 8
    return {"bytes": b, "flops": 0}


def _exact_mlp(w, x, t=None):
    """The 16-64-64-2 ReLU network on weights rounded to bfloat16, and the mean-squared-error gradient."""
    sizes = [(learn.NIN, 64), (64,), (64, 64), (64,), (64, learn.NOUT), (learn.NOUT,)]
    parts = torch.from_numpy(w).bfloat16().double().split([math.prod(s) for s in sizes])
    w1, b1, w2, b2, w3, b3 = (p.reshape(s).clone().requires_grad_(t is not None) for p, s in zip(parts, sizes))
    y = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2) @ w3 + b3
    if t is None:
        return y
    loss = ((y - t) ** 2).mean()
    grads = torch.autograd.grad(loss, (w1, b1, w2, b2, w3, b3))
    return loss.item(), torch.cat([g.reshape(-1) for g in grads])


def _exact_features(case, hg):
    """The 16 features of every root edge of a labeled query, in root order, from their definitions."""
    k, edges = SHAPES[case["pattern"]]
    lab = _pattern_labels(case)
    pdeg = [sum(v in e for e in edges) for v in range(k)]
    n, rp, dst = hg.n, hg.rowptr.astype(np.int64), hg.colidx.astype(np.int64)
    deg, labels = np.diff(rp), hg.labels.astype(np.int64)
    src = np.repeat(np.arange(n), deg)
    ldst = labels[dst]

    def total(weights):
        return np.bincount(src, weights=weights, minlength=n)

    maxnbr = np.zeros(n, dtype=np.int64)
    some = np.nonzero(deg)[0]
    maxnbr[some] = np.maximum.reduceat(deg[dst], rp[:-1][some])
    match2, next3 = total(ldst == lab[2]), total(ldst == lab[3])
    pairs, two_hop = total((ldst == lab[2]) * next3[dst]), total(deg[dst])
    hist = np.bincount(src * 8 + (ldst & 7), minlength=8 * n).reshape(n, 8)
    bucket = np.minimum(np.floor(np.log2(1.0 + deg) * 4).astype(np.int64), 255)
    rank = np.cumsum(np.bincount(bucket, minlength=256))[bucket] / n
    keep = ((labels[src] == lab[0]) & (ldst == lab[1]) & (deg[src] >= pdeg[0]) & (deg[dst] >= pdeg[1])
            & (maxnbr[dst] >= pdeg[2]))
    r, c = src[keep], dst[keep]
    d1 = deg[c].astype(np.float64)
    cols = [np.log2(1.0 + deg[r]), np.log2(1.0 + d1), np.log2(1 + match2[c]), np.log2(1 + pairs[c]),
            np.log2(1 + two_hop[c]), np.log2(1.0 + maxnbr[c]), rank[c]]
    cols += [hist[c, q] / d1 for q in range(8)] + [match2[c] / d1]
    out = np.zeros((_root_cap(case), learn.NIN))
    out[:len(r)] = np.stack(cols, axis=1)
    return torch.from_numpy(out)


def exact(case, seed):
    if case["do"] == "features":
        return _exact_features(case, _host_graph(case, seed))
    if "samples" not in case:
        return None  # counts, set operations, root lists: whole numbers
    w, mu, sd, x, t = _model_data(case, seed)
    if case["do"] == "predict":
        y = _exact_mlp(w, (x.double() - torch.from_numpy(mu).double()) / torch.from_numpy(sd).double())
        return y * torch.tensor([3.0, 2.0], dtype=torch.float64) + torch.tensor([15.0, 6.0], dtype=torch.float64)
    loss, grad = _exact_mlp(w, x.double(), t.double())
    return {"loss": loss, "grad": grad}
