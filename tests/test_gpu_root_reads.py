"""Per-root adjacency-list reads (a training target of the learned scheduler): what the level-by-level search reads,
whatever scheme a launch takes and however its ranges are cut."""
import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    hg = pm.gen_chung_lu(600, 9000, gamma=2.3, i0=5.0, max_w=90.0, seed=11)
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg)
    yield ctx, g
    g.close()
    ctx.close()


def reads(ctx, g, p, **kw):
    out = torch.zeros(max(1, ctx.count_roots(g, p)), device="cuda")
    torch.cuda.synchronize()
    counts, _ = ctx.match(g, [p], root_reads_ptr=out.data_ptr(), timeout_ms=60000, **kw)
    return counts[0], out.cpu().numpy()


@pytest.mark.parametrize("k", [5, 6, 7])
@pytest.mark.parametrize("kw", [dict(), dict(split_level1=2, chunk=1), dict(split_level1=-1, chunk=500),
                                dict(lane_subtree_max=512)], ids=str)
def test_cliques_read_what_the_search_reads(setup, k, kw):
    ctx, g = setup
    p = pm.PatternPreprocessor(text=P.to_g(*P.clique(k)), labeled=False)
    want = reads(ctx, g, p, lane_subtree_max=-1)
    got = reads(ctx, g, p, **kw)
    assert got[0] == want[0] and want[1].sum() > len(want[1])
    assert np.array_equal(got[1], want[1])
