"""Placing a graph: what it holds per vertex is one allocation with its rows, given back with them; graphs from the host
and from device arrays, of any size and parity, give the same root lists and counts."""
import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = pm.Context(0)
    yield c
    c.close()


def hubs(n):
    """Two vertices adjacent to all n others, which form a path (lists long enough for bit rows from n = 64 on)."""
    rows = [sorted({v for v in (i - 1, i + 1) if 0 <= v < n} | {n, n + 1}) for i in range(n)]
    rows += [list(range(n)) + [n + 1], list(range(n + 1))]
    return pm.HostGraph(np.cumsum([0] + [len(r) for r in rows]).astype(np.uint64),
                        np.concatenate([np.array(r, dtype=np.int32) for r in rows]))


@pytest.mark.parametrize("n", [1, 2, 31, 62, 63, 64, 65, 200, 1001])
@pytest.mark.parametrize("labeled", [False, True])
def test_host_and_device_arrays(ctx, n, labeled):
    hg = hubs(n)
    labels = (np.arange(hg.n) % 3).astype(np.uint32)
    host = pm.GraphPreprocessor.from_host(pm.HostGraph(hg.rowptr, hg.colidx, labels if labeled else None), labeled=labeled)
    rp, ci = torch.from_numpy(hg.rowptr.astype(np.int64)).cuda(), torch.from_numpy(hg.colidx).cuda()
    lb = torch.from_numpy(labels.astype(np.uint8)).cuda() if labeled else None
    dev = pm.GraphPreprocessor.from_device(hg.n, hg.n_adj, hg.max_degree, rp.data_ptr(), ci.data_ptr(),
                                           lb.data_ptr() if labeled else None)
    for k, e in (P.clique(4), P.clique(5), P.cycle(5), P.house()):
        p = pm.PatternPreprocessor(text=P.to_g(k, e, [i % 3 for i in range(k)] if labeled else None), labeled=labeled)
        assert np.array_equal(ctx.roots(host, p), ctx.roots(dev, p))
        (a, sa), (b, sb) = (ctx.match(g, [p], timeout_ms=60000) for g in (host, dev))
        assert (a, sa["set_ops"], sa["alg_bytes"]) == (b, sb["set_ops"], sb["alg_bytes"])
    host.close()
    dev.close()


@pytest.mark.parametrize("kw", [dict(), dict(labeled=True), dict(paged=True, page_bytes=4096, frame_pool_bytes=1 << 20)],
                         ids=str)
def test_memory_is_given_back(kw):
    hg = pm.gen_chung_lu(100_000, 600_000, seed=2)
    hg = pm.HostGraph(hg.rowptr, hg.colidx, pm.gen_labels(hg.n, 4, 1))
    pm.GraphPreprocessor.from_host(hg, **kw).close()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        pm.GraphPreprocessor.from_host(hg, **kw).close()
    assert torch.cuda.mem_get_info()[0] == free
