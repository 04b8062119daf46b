"""Cliques in bit sets against the plain search: counts, set operations and algorithmic bytes, for common
neighbourhoods at the edges of the word, row and matrix sizes."""
import numpy as np
import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def two_hubs(m, per, seed):
    """Vertices m and m+1 adjacent to each other and to all of 0..m-1, which form a random graph of `per`
    neighbours each."""
    r = np.random.default_rng(seed)
    k = min(m * per // 2, m * (m - 1) // 2)
    e = {(i, h) for i in range(m) for h in (m, m + 1)} | {(m, m + 1)}
    e |= {(int(a), int(b)) for a, b in r.integers(0, m, (k, 2)) if a < b}
    rows = [[] for _ in range(m + 2)]
    for a, b in e:
        rows[a].append(b)
        rows[b].append(a)
    rp = np.cumsum([0] + [len(x) for x in rows]).astype(np.uint64)
    return pm.HostGraph(rp, np.concatenate([np.sort(x) for x in rows]).astype(np.int32))


@pytest.fixture(scope="module")
def ctx():
    c = pm.Context(0)
    yield c
    c.close()


def both(ctx, hg, k, **kw):
    g = pm.GraphPreprocessor.from_host(hg, labeled=False)
    p = pm.PatternPreprocessor(text=P.to_g(*P.clique(k)), labeled=False)
    out = []
    for lane in (0, -1):  # bit sets, and never a lane or bit-set scheme
        c, st = ctx.match(g, [p], lane_subtree_max=lane, timeout_ms=60000, **kw)
        out.append((c[0], st["n_roots"], st["set_ops"], st["alg_bytes"]))
    g.close()
    return out


@pytest.mark.parametrize("k", [5, 6, 7])
@pytest.mark.parametrize("m", [1, 3, 31, 32, 33, 64, 65, 128, 129, 512, 513, 1023, 1024, 1025])
def test_two_hubs(ctx, m, k):
    a, b = both(ctx, two_hubs(m, min(m, 24), 7 * m + k), k)
    assert a == b


@pytest.mark.parametrize("n,k", [(5, 5), (34, 5), (35, 6), (66, 5), (40, 7)])
def test_complete_graph(ctx, n, k):
    rp = (np.arange(n + 1) * (n - 1)).astype(np.uint64)
    ci = np.concatenate([[j for j in range(n) if j != i] for i in range(n)]).astype(np.int32)
    a, b = both(ctx, pm.HostGraph(rp, ci), k)
    assert a == b
    want = 1
    for i in range(k):
        want *= n - i
    assert a[0] == want


def test_matrix_beyond_the_arena(ctx):
    """A matrix that does not fit the warp's arena: the level below takes over."""
    a, b = both(ctx, two_hubs(300, 40, 3), 6, own_arena_words=2048)
    assert a == b
