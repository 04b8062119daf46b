"""The last two levels in one pass against the level-by-level search: counts, set operations, algorithmic bytes and
per-root counts, over the plans it takes (every kind of main slot and last slot), truncation, residency, list
lengths around a tile, value tables that are too small, and graphs whose entries have no reverse."""
import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu

SHAPES = {"C5": P.cycle(5), "C6": P.cycle(6), "C7": P.cycle(7), "P4": P.path(4), "P5": P.path(5), "P6": P.path(6), "P7": P.path(7), "house": P.house(),
          "house_tail": P.house_tail(1), "house_tail2": P.house_tail(2), "C4_tail": P.cycle_tail(4, 1),
          "C4_tail2": P.cycle_tail(4, 2), "C5_tail2": P.cycle_tail(5, 2), "C6_tail": P.cycle_tail(6, 1),
          "S5": P.star(5)}


@pytest.fixture(scope="module")
def ctx():
    c = pm.Context(0)
    yield c
    c.close()


def runs(ctx, hg, shape, labels, n_labels=0, paged=False, **kw):
    """(counts, stats, per-root counts) in one pass and level by level."""
    labeled = n_labels > 0
    k, e = SHAPES[shape]
    p = pm.PatternPreprocessor(text=P.to_g(k, e, P.seeded_labels(k, n_labels, 5) if labeled else None), labeled=labeled)
    kwg = dict(paged=True, page_bytes=4096, frame_pool_bytes=64 << 10, static_pool_bytes=16 << 10) if paged else {}
    g = pm.GraphPreprocessor.from_host(pm.HostGraph(hg.rowptr, hg.colidx, labels), labeled=labeled, **kwg)
    out = []
    for leaf in (0, 1):
        per = torch.zeros(max(1, ctx.count_roots(g, p)), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        c, st = ctx.match(g, [p], leaf_per_lane=leaf, root_counts_ptr=per.data_ptr(), timeout_ms=60000, **kw)
        out.append((c[0], st["n_roots"], st["set_ops"], st["alg_bytes"], per.cpu().numpy()))
    g.close()
    return out


def same(a, b):
    assert a[:4] == b[:4]
    assert np.array_equal(a[4], b[4])


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("truncate", [0, 5])
def test_unlabeled(ctx, shape, truncate):
    same(*runs(ctx, pm.gen_chung_lu(150, 420, seed=3), shape, None, truncate=truncate))


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("truncate,paged", [(0, False), (3, False), (0, True)])
def test_labeled(ctx, shape, truncate, paged):
    hg = pm.gen_rmat(600, 4000, seed=4)
    same(*runs(ctx, hg, shape, pm.gen_labels(hg.n, 4, 9), 4, paged=paged, truncate=truncate))


@pytest.mark.parametrize("n", [31, 32, 33, 127, 128, 129, 160])
@pytest.mark.parametrize("shape", ["C5", "house", "C4_tail"])
def test_list_lengths_around_a_tile(ctx, n, shape):
    """A ring of n vertices with two hubs adjacent to all of it: lists of 4 and of about n elements."""
    rows = [sorted({(i - 1) % n, (i + 1) % n, n, n + 1}) for i in range(n)]
    rows += [list(range(n)) + [n + 1], list(range(n + 1))]
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.uint64)
    same(*runs(ctx, pm.HostGraph(rp, np.concatenate(rows).astype(np.int32)), shape, None))


@pytest.mark.parametrize("shape", ["C5", "C6"])
def test_ids_beyond_the_bitmap_and_the_table(ctx, shape):
    """Ids spread past 16,384: the filter instead of the bitmap, table entries shared by several vertices."""
    small = pm.gen_chung_lu(300, 900, seed=6)
    at = np.sort(np.random.default_rng(7).choice(70_000, small.n, replace=False))
    deg = np.zeros(70_000, dtype=np.int64)
    deg[at] = np.diff(small.rowptr.astype(np.int64))
    hg = pm.HostGraph(np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64), at[small.colidx].astype(np.int32))
    a = runs(ctx, hg, shape, None)
    same(*a)
    assert a[0][:3] == runs(ctx, small, shape, None)[0][:3]


@pytest.mark.parametrize("shape", ["C5", "P5", "house", "C4_tail"])
def test_entries_without_their_reverse(ctx, shape):
    """Not an undirected graph: nothing is taken from one list about another."""
    hg = pm.gen_chung_lu(120, 500, seed=8)
    keep = np.random.default_rng(1).random(hg.n_adj) < 0.8
    rp = np.concatenate([[0], np.cumsum(keep)])[hg.rowptr.astype(np.int64)]
    same(*runs(ctx, pm.HostGraph(rp.astype(np.uint64), hg.colidx[keep]), shape, None))


def test_one_context_many_graphs(ctx):
    """The value tables outlive a call: other graphs, plans and launch shapes on the same context."""
    for seed, shape, wpb in ((1, "C5", 8), (2, "C5", 8), (1, "C6", 4), (3, "C5", 16), (1, "C5", 8)):
        hg = pm.gen_chung_lu(100 + 30 * seed, 400, seed=seed)
        same(*runs(ctx, hg, shape, None, warps_per_block=wpb))


@pytest.mark.parametrize("shape", [P.star(6), P.star(7), P.house_tail(1), P.house_tail(2)])
@pytest.mark.parametrize("truncate,paged", [(0, False), (4, False), (0, True)])
def test_levels_of_copies(ctx, shape, truncate, paged):
    """One candidate searched for all where the next level only copies: against the oracle, also when pieces of the
    search change hands."""
    import os
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
    import pm_oracle as orc
    hg = pm.gen_rmat(300, 1500, seed=2)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, 3, 4))
    k, e = shape
    text = P.to_g(k, e, P.seeded_labels(k, 3, 8))
    og, op = orc.Graph(hg.rowptr, hg.colidx, hg.labels), orc.plan(text, True)
    want, st0 = orc.count(og, op, orc.roots(og, op), truncate=truncate)
    kw = dict(paged=True, page_bytes=4096, frame_pool_bytes=64 << 10) if paged else {}
    g = pm.GraphPreprocessor.from_host(hg, labeled=True, **kw)
    p = pm.PatternPreprocessor(text=text, labeled=True)
    for split in (0, 2, -1):
        c, st = ctx.match(g, [p], truncate=truncate, split_level1=split, timeout_ms=60000)
        assert (c[0], st["set_ops"], st["alg_bytes"]) == (want, st0["set_ops"], st0["alg_bytes"])
    g.close()


@pytest.mark.parametrize("shape", ["C5", "house", "C4_tail", "house_tail"])
def test_elements_that_come_twice(ctx, shape):
    """A list that holds an element twice is no simple graph's: bit rows and what one list says of another are not
    used, and both ways count alike."""
    hg = pm.gen_chung_lu(120, 500, seed=9)
    src = np.repeat(np.arange(hg.n), np.diff(hg.rowptr.astype(np.int64)))
    e = [(int(a), int(b)) for a, b in zip(src, hg.colidx)]
    e += [x for a, b in e if a < b and (a + b) % 7 == 0 for x in ((a, b), (b, a))]
    e.sort()
    rp = np.concatenate([[0], np.cumsum(np.bincount([a for a, _ in e], minlength=hg.n))])
    same(*runs(ctx, pm.HostGraph(rp.astype(np.uint64), np.array([b for _, b in e], dtype=np.int32)), shape, None))
