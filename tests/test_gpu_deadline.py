"""A launch past its limit ends soon after it, whatever its warps are in, and leaves the context usable.  (The graphs are
skewed: hubs' lists of tens of thousands of elements, where one warp's pass over them is longest.)"""
import time

import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu

LIMIT_MS = 2
# Between two looks at the clock a warp walks at most some thousands of elements, or the lists of as many: well under
# the 136 ms that a pass over 32 hubs' lists took.  The bound is on the host's clock, root filter included.
BOUND_MS = 60


def expired(ctx, g, p):
    """Milliseconds of a call that runs into its limit."""
    t0 = time.perf_counter()
    with pytest.raises(pm.PmError) as e:
        ctx.match(g, [p], timeout_ms=LIMIT_MS)
    ms = (time.perf_counter() - t0) * 1e3
    assert e.value.status == pm.PM_ERR_TIMEOUT
    return ms


@pytest.mark.parametrize("labels,shapes", [(0, [P.cycle(5), P.cycle(6), P.cycle(7), P.house(), P.house_tail(2), P.path(5),
                                                P.path(6), P.cycle_tail(4, 1), P.clique(7)]),
                                           (4, [P.cycle(5), P.cycle(6), P.cycle(7), P.house_tail(2), P.clique(6)])],
                         ids=["unlabeled", "labeled"])
def test_launches_past_their_limit(labels, shapes):
    hg = pm.gen_rmat(262_144, 4_194_304, seed=3, device=0)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, labels, 5) if labels else None)
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg, labeled=labels > 0)
    small = pm.GraphPreprocessor.from_host(pm.gen_chung_lu(400, 2000, seed=1))
    ps = pm.PatternPreprocessor(text=P.to_g(*P.house()), labeled=False)
    want = ctx.match(small, [ps])[0]
    for k, e in shapes:
        p = pm.PatternPreprocessor(text=P.to_g(k, e, P.seeded_labels(k, labels, 202) if labels else None),
                                   labeled=labels > 0)
        ctx.match(g, [p], root_begin=0, root_end=0)  # (buffers, and the kernel's first load)
        assert min(expired(ctx, g, p) for _ in range(3)) < BOUND_MS, (k, e)
        assert ctx.match(small, [ps])[0] == want
    g.close()
    small.close()
    ctx.close()


def test_prepared_query_past_its_limit():
    hg = pm.gen_rmat(32_768, 524_288, seed=3, device=0)
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(hg)
    p = pm.PatternPreprocessor(text=P.to_g(*P.cycle(7)), labeled=False)
    q = ctx.prepare(g, [p], timeout_ms=LIMIT_MS)
    for _ in range(2):
        with pytest.raises(pm.PmError) as e:
            q.run()
        assert e.value.status == pm.PM_ERR_TIMEOUT
    q.close()
    a = ctx.match(g, [p], root_begin=0, root_end=16)
    assert a[0] == ctx.match(g, [p], root_begin=0, root_end=16)[0] and a[1]["device_status"] == 0
    g.close()
    ctx.close()
