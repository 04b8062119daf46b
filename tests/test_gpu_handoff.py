"""Work hand-off between warps: every root processed once whatever the pop size, the number of warps and the
share of them that start without roots (tickets, pieces and the end of the launch)."""
import os

import numpy as np
import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu

GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "graphs")


@pytest.fixture(scope="module")
def setup():
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(GOLD), "..", "..", "oracle"))
    import pm_oracle as orc
    hg = pm.HostGraph.read(os.path.join(GOLD, "cl400"), labeled=True)
    text = P.to_g(*P.house())
    og, p = orc.Graph(hg.rowptr, hg.colidx, None), orc.plan(text, False)
    count, st = orc.count(og, p, orc.roots(og, p))
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg, labeled=False)
    yield ctx, g, pm.PatternPreprocessor(text=text, labeled=False), count * p.multiplicity, st["set_ops"]
    g.close()
    ctx.close()


@pytest.mark.parametrize("wpb,bps", [(1, 1), (8, 1), (8, 0), (16, 0)])
@pytest.mark.parametrize("chunk", [0, 1, 3, 17, 4096])
def test_every_root_once(setup, chunk, wpb, bps):
    ctx, g, p, want, set_ops = setup
    got, st = ctx.match(g, [p], chunk=chunk, warps_per_block=wpb, blocks_per_sm=bps, timeout_ms=60000)
    assert got[0] == want and st["set_ops"] == set_ops


@pytest.mark.parametrize("chunk", [0, 5])
@pytest.mark.parametrize("shards", [2, 3, 64, 1000])
def test_shards_partition_the_roots(setup, chunk, shards):
    ctx, g, p, want, set_ops = setup
    runs = [ctx.match(g, [p], chunk=chunk, shard_rank=r, shard_count=shards, timeout_ms=60000)
            for r in range(min(shards, 80))]
    n = ctx.count_roots(g, p)
    if shards <= 80:
        assert sum(c[0] for c, _ in runs) == want and sum(s["set_ops"] for _, s in runs) == set_ops
    # a shard's roots are its units of `chunk` (16 by default) roots, whatever the pop size
    unit = chunk or 16
    mine = [int(np.sum((np.arange(n) // unit) % shards == r)) for r in range(len(runs))]
    assert [s["n_roots"] for _, s in runs] == mine


@pytest.mark.parametrize("roots", [0, 1, 2, 33])
def test_few_roots_many_warps(setup, roots):
    ctx, g, p, _, _ = setup
    a, sa = ctx.match(g, [p], root_begin=0, root_end=roots, timeout_ms=60000)
    b, sb = ctx.match(g, [p], root_begin=0, root_end=roots, split_level1=-1, timeout_ms=60000)
    assert a == b and sa["set_ops"] == sb["set_ops"] and sa["n_roots"] == roots
