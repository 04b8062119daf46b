"""Passes over all adjacency lists (placement, root filter, root features): list lengths around a tile and around
the length from which a block takes a list, against plain numpy."""
import numpy as np
import pytest

import pumatch_b200 as pm
from pumatch_b200 import learn
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def star_forest(lengths, seed):
    """One hub per length, each adjacent to that many of a shared pool of vertices, and the pool a ring."""
    pool = max(lengths) + 3
    n = pool + len(lengths)
    r = np.random.default_rng(seed)
    e = {(i, (i + 1) % pool) for i in range(pool)}
    for k, m in enumerate(lengths):
        e |= {(int(i), pool + k) for i in r.choice(pool, m, replace=False)}
    rows = [[] for _ in range(n)]
    for a, b in e:
        rows[a].append(b)
        rows[b].append(a)
    rp = np.cumsum([0] + [len(x) for x in rows]).astype(np.uint64)
    return pm.HostGraph(rp, np.concatenate([np.sort(x) for x in rows]).astype(np.int32))


LENGTHS = [1, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 1535, 1536, 1537, 5000]


@pytest.fixture(scope="module")
def case():
    hg = star_forest(LENGTHS, 3)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, 3, 5))
    ctx = pm.Context(0)
    yield ctx, hg
    ctx.close()


def arrays(hg):
    rp = hg.rowptr.astype(np.int64)
    deg = np.diff(rp)
    src, dst = np.repeat(np.arange(hg.n), deg), hg.colidx.astype(np.int64)
    nbr = np.zeros(hg.n, dtype=np.int64)
    np.maximum.at(nbr, src, deg[dst])
    return rp, deg, src, dst, nbr


@pytest.mark.parametrize("labeled", [False, True])
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("shape", [P.star(6), P.cycle(4), P.path(4)])
def test_root_filter(case, shape, labeled, paged):
    ctx, hg = case
    rp, deg, src, dst, nbr = arrays(hg)
    labs = [0, 1, 2, 0, 1, 2][:shape[0]]
    p = pm.PatternPreprocessor(text=P.to_g(*shape, labs if labeled else None), labeled=labeled)
    kw = dict(paged=True, page_bytes=4096, frame_pool_bytes=64 << 10) if paged else {}
    g = pm.GraphPreprocessor.from_host(hg, labeled=labeled, **kw)
    d = p.describe()["degree"]
    keep = (deg[src] >= d[0]) & (deg[dst] >= d[1]) & (nbr[dst] >= d[2])
    if labeled:
        keep &= (hg.labels[src] == labs[0]) & (hg.labels[dst] == labs[1])
    elif p.describe()["partial"][0] == 1:
        keep &= src > dst
    got = ctx.roots(g, p)
    assert np.array_equal(got, np.stack([src[keep], dst[keep]], axis=1))
    g.close()


def test_label_groups_by_counts(case):
    """Every list's label groups, through the counts of two-edge paths by label (a wrong group would change one)."""
    ctx, hg = case
    rp, deg, src, dst, nbr = arrays(hg)
    g = pm.GraphPreprocessor.from_host(hg, labeled=True)
    for l2 in range(3):
        p = pm.PatternPreprocessor(text=P.to_g(*P.path(3), [0, 1, l2]), labeled=True)
        per = np.bincount(src, weights=hg.labels[dst] == l2, minlength=hg.n).astype(np.int64)
        keep = (hg.labels[src] == 0) & (hg.labels[dst] == 1) & (deg[dst] >= 2)
        counts, _ = ctx.match(g, [p], timeout_ms=60000)
        assert counts[0] == per[dst[keep]].sum()
    g.close()


def test_root_features(case):
    ctx, hg = case
    rp, deg, src, dst, nbr = arrays(hg)
    p = pm.PatternPreprocessor(text=P.to_g(*P.path(4), [0, 1, 2, 0]), labeled=True)
    g = pm.GraphPreprocessor.from_host(hg, labeled=True)
    x = learn.root_features(ctx, g, p).cpu().numpy().astype(np.float64)
    roots = ctx.roots(g, p)
    ldst = hg.labels[dst].astype(np.int64)
    tot = lambda w: np.bincount(src, weights=w, minlength=hg.n)  # noqa: E731
    m2, n0 = tot(ldst == 2), tot(ldst == 0)
    c = roots[:, 1]
    want = {0: np.log2(1 + deg[roots[:, 0]]), 1: np.log2(1 + deg[c]), 2: np.log2(1 + m2[c]),
            3: np.log2(1 + tot((ldst == 2) * n0[dst])[c]), 4: np.log2(1 + tot(deg[dst])[c]), 5: np.log2(1 + nbr[c]),
            15: m2[c] / deg[c]}
    want |= {7 + k: tot((ldst & 7) == k)[c] / deg[c] for k in range(8)}
    for k, w in want.items():  # whole sums, one logarithm or division: a few units in the last place
        assert np.allclose(x[:, k], w, rtol=4 * 2.0 ** -23, atol=1e-7), k
    g.close()
