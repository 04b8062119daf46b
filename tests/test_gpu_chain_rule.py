"""Tables for a plan's chain are worked out for a whole graph in each launch: a launch of few roots does without."""
import numpy as np
import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def test_few_roots_of_a_large_graph():
    hg = pm.gen_rmat(4_000_000, 32_000_000, seed=5, device=0)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, 8, 5))
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg, labeled=True)
    p = pm.PatternPreprocessor(text=P.to_g(*P.path(4), P.seeded_labels(4, 8, 202)), labeled=True)

    def run(**kw):
        runs = [ctx.match(g, [p], timeout_ms=60000, **kw) for _ in range(4)]
        return runs[0][0][0], runs[0][1]["set_ops"], min(st["kernel_ms"] for _, st in runs)

    whole = run()
    few = run(root_begin=1000, root_end=1016)
    assert few[2] < 0.5 * whole[2]  # no pass over the graph
    # the same roots' share with and without tables
    n = ctx.count_roots(g, p)
    parts = [run(root_begin=b, root_end=b + 16)[:2] for b in (1000, n // 2)]
    searched = [run(root_begin=b, root_end=b + 16, leaf_per_lane=1)[:2] for b in (1000, n // 2)]
    assert parts == searched and parts[0] == few[:2]
    g.close()
    ctx.close()


@pytest.mark.parametrize("shape", [P.path(4), P.path(5), P.path(6), P.cycle_tail(4, 2), P.cycle_tail(5, 2)])
def test_counts_on_either_side(shape):
    """Root ranges from one root to all of them: with tables, without, and one after the other."""
    hg = pm.gen_rmat(60_000, 400_000, seed=6, device=0)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, 4, 7))
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg, labeled=True)
    k, e = shape
    p = pm.PatternPreprocessor(text=P.to_g(k, e, P.seeded_labels(k, 4, 9)), labeled=True)
    n = ctx.count_roots(g, p)
    cuts = [0, 1, 17, 300, n // 2, n]
    total = np.zeros(3, dtype=object)
    for b, e in zip(cuts, cuts[1:]):
        c, st = ctx.match(g, [p], root_begin=b, root_end=e, timeout_ms=60000)
        total += np.array([c[0], st["set_ops"], st["alg_bytes"]], dtype=object)
    c, st = ctx.match(g, [p], timeout_ms=60000)
    assert list(total) == [c[0], st["set_ops"], st["alg_bytes"]]
    g.close()
    ctx.close()
