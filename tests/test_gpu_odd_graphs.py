"""Graphs that are not simple and undirected -- vertices in their own lists, elements that come twice, entries without
their reverse -- with hubs whose lists are long enough for bit rows: counts, set operations and algorithmic bytes
against a host search written here from the definition of a plan's set operations."""
import numpy as np
import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu

SHAPES = {"P4": P.path(4), "house": P.house(), "house_tail": P.house_tail(1), "C4_tail": P.cycle_tail(4, 1),
          "C4": P.cycle(4), "C5": P.cycle(5), "K4": P.clique(4), "K5": P.clique(5), "K6": P.clique(6)}


def entries(n, per, seed):
    """Both directions of a random graph on n vertices with two hubs adjacent to all of it, and how many vertices."""
    r = np.random.default_rng(seed)
    e = {(i, h) for i in range(n) for h in (n, n + 1)} | {(n, n + 1)}
    e |= {(int(min(a, b)), int(max(a, b))) for a, b in r.integers(0, n, (n * per // 2, 2)) if a != b}
    return sorted(e | {(b, a) for a, b in e}), n + 2


def host_graph(e, n, labels=None):
    e = sorted(e)
    rp = np.concatenate([[0], np.cumsum(np.bincount([a for a, _ in e], minlength=n))]).astype(np.uint64)
    return pm.HostGraph(rp, np.array([b for _, b in e], dtype=np.int32), labels)


class Search:
    """A plan's search, one set operation after the other: N(v_L) (fresh), N(v_L) met with the parent slot, or the
    parent slot (copy), the first operand cut at the plan's bound, less the path vertices (fresh) or v_L (copy) when
    unlabeled, by label else, at most T long.  Of the last level's fresh set or copy only the size counts, less one for
    each of v_0 .. v_{n-3} (fresh) or for v_{n-2} (copy) in it, however often it is there."""

    def __init__(self, hg, p, truncate):
        self.d, self.T = p.describe(), truncate
        rp = hg.rowptr.astype(np.int64)
        self.adj = [[int(x) for x in hg.colidx[rp[v]:rp[v + 1]]] for v in range(hg.n)]
        self.labels = None if hg.labels is None else [int(x) for x in hg.labels]
        self.count = self.ops = self.bytes = 0

    def slot(self, s, L, path, slots, last):
        d, T = self.d, self.T
        op, labeled = d["set_ops"][s], bool(d["labeled"])
        par, fresh, meet = op & 31, bool(op & 0x20), bool(op & 0x40)
        up = slots[par] if L > 1 else self.adj[path[0]]
        A = self.adj[path[L]] if fresh or meet else up
        B = up if meet else []
        main = s == d["level_begin"][L]
        if not labeled and d["partial"][s]:
            vs = [path[j] for j in range(L + 1) if d["partial"][s] >> j & 1]
            if vs:
                ub = min(vs) if main else max(vs)
                A = A[:int(np.searchsorted(A, ub))]
        if labeled:
            member = set(B)
            out = [x for x in A if d["slot_labels"][s] >> self.labels[x] & 1 and (not meet or x in member)]
        elif meet:
            member = set(B)
            out = [x for x in A if x in member]
        elif fresh and last:
            out = A[:T] if T else A
            size = len(out) - sum(v in out for v in path[:L])
        elif fresh:
            out = [x for x in (A[:T] if T else A) if x not in path]
        elif last:
            out, size = A, len(A) - (path[L] in A)
            size = min(size, T) if T else size
        else:
            out = [x for x in A if x != path[L]]
        if labeled or meet or not last:
            out = out[:T] if T else out
            size = len(out)
        self.ops += 1
        self.bytes += 4 * (len(A) + len(B) + size) + (len(A) if labeled else 0)
        return size if last else out

    def below(self, L, path, slots):
        d, n = self.d, self.d["nnodes"]
        if L == n - 2:
            self.count += self.slot(d["level_begin"][L], L, path, slots, True)
            return
        slots = dict(slots)
        for s in range(d["level_begin"][L], d["level_begin"][L + 1]):
            slots[s] = self.slot(s, L, path, slots, False)
        for v in slots[d["level_begin"][L]]:
            self.below(L + 1, path + [v], slots)

    def run(self, roots):
        for a, b in roots:
            self.bytes += 8
            self.below(1, [int(a), int(b)], {})
        return self.count * (1 if self.d["labeled"] else self.d["multiplicity"]), self.ops, self.bytes


@pytest.fixture(scope="module")
def ctx():
    c = pm.Context(0)
    yield c
    c.close()


def check(ctx, hg, shape, labeled, truncate, paged=False, **kw):
    k, e = SHAPES[shape]
    p = pm.PatternPreprocessor(text=P.to_g(k, e, P.seeded_labels(k, 3, 5) if labeled else None), labeled=labeled)
    pool = dict(paged=True, page_bytes=4096, frame_pool_bytes=64 << 10) if paged else {}
    g = pm.GraphPreprocessor.from_host(hg, labeled=labeled, **pool)
    try:
        got, st = ctx.match(g, [p], truncate=truncate, timeout_ms=60000, **kw)
        want = Search(hg, p, truncate).run(ctx.roots(g, p))
    finally:
        g.close()
    assert (got[0], st["set_ops"], st["alg_bytes"]) == want


@pytest.mark.parametrize("truncate", [0, 5])
@pytest.mark.parametrize("shape", ["P4", "house", "house_tail", "C4_tail", "C5", "K4", "K5"])
@pytest.mark.parametrize("step", [0, 3])
def test_vertices_in_their_own_lists(ctx, shape, step, truncate):
    """Both hubs, alone or with every third vertex."""
    e, n = entries(90, 4, 1)
    loops = [(v, v) for v in (range(0, n - 2, step) if step else [])] + [(n - 2, n - 2), (n - 1, n - 1)]
    check(ctx, host_graph(e + loops, n), shape, False, truncate)


@pytest.mark.parametrize("truncate", [0, 5])
@pytest.mark.parametrize("shape", ["P4", "C4", "C5", "house", "house_tail", "C4_tail", "K5"])
@pytest.mark.parametrize("paged", [False, True])
def test_labeled_elements_that_come_twice(ctx, shape, truncate, paged):
    """A list that holds an element twice can meet a set of at most T elements in more than T."""
    e, n = entries(90, 4, 1)
    e += [x for a, b in e if a < b and (a * 7 + b) % 5 == 0 for x in ((a, b), (b, a))]
    labels = (np.arange(n) * 7 % 5 % 3).astype(np.uint32)
    check(ctx, host_graph(e, n, labels), shape, True, truncate, paged)


@pytest.mark.parametrize("truncate", [0, 5])
@pytest.mark.parametrize("shape", ["K5", "K6"])
@pytest.mark.parametrize("lane", [0, 512])
def test_cliques_of_elements_that_come_twice(ctx, shape, truncate, lane):
    """More of a doubled list is in the parent set than the set has elements: the scheme of one candidate per lane,
    whose lanes have room for the set, leaves the node to the search."""
    e, n = entries(70, 12, 3)
    e += [x for a, b in e if a < b and (a + b) % 3 for x in ((a, b), (b, a))]
    check(ctx, host_graph(e, n), shape, False, truncate, lane_subtree_max=lane)


@pytest.mark.parametrize("shape,labeled", [("K5", False), ("K6", False), ("house_tail", False), ("house", True), ("K5", True)])
@pytest.mark.parametrize("words", [1, 80, 200])
def test_small_arenas_and_elements_that_come_twice(ctx, shape, labeled, words):
    """A doubled list can meet a set in more elements than the set has: the arena is asked for room for all of them
    (a warp whose own is too small borrows a larger one)."""
    e, n = entries(70, 12, 3)
    e += [x for a, b in e if a < b and (a + b) % 3 for x in ((a, b), (b, a))]
    labels = (np.arange(n) * 7 % 5 % 3).astype(np.uint32) if labeled else None
    check(ctx, host_graph(e, n, labels), shape, labeled, 0, lane_subtree_max=-1, own_arena_words=words)


@pytest.mark.parametrize("truncate", [0, 5])
@pytest.mark.parametrize("shape", ["P4", "house", "house_tail", "C4_tail", "C5"])
def test_elements_that_come_twice(ctx, shape, truncate):
    e, n = entries(90, 4, 1)
    e += [x for a, b in e if a < b and (a * 7 + b) % 5 == 0 for x in ((a, b), (b, a))]
    check(ctx, host_graph(e, n), shape, False, truncate)


@pytest.mark.parametrize("truncate", [0, 5])
@pytest.mark.parametrize("shape", ["P4", "house", "house_tail", "C4_tail", "C5", "K4", "K5"])
@pytest.mark.parametrize("labeled", [False, True])
def test_entries_without_their_reverse(ctx, shape, labeled, truncate):
    e, n = entries(90, 4, 1)
    e = [x for x in e if (x[0] * 31 + x[1] * 17) % 9]
    labels = (np.arange(n) * 7 % 5 % 3).astype(np.uint32) if labeled else None
    check(ctx, host_graph(e, n, labels), shape, labeled, truncate)
