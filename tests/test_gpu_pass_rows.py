"""Passes over the last two levels that take a part of their candidates, or of one list: lists around and beyond what a
pass walks, against the level-by-level search (counts, set operations, algorithmic bytes, per-root counts and reads)."""
import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def hubs(n):
    """A ring of n vertices and three hubs: two adjacent to all of it, one to every fifth vertex."""
    rows = [sorted({(i - 1) % n, (i + 1) % n, n, n + 1} | ({n + 2} if i % 5 == 0 else set())) for i in range(n)]
    rows += [list(range(n)) + [n + 1], list(range(n + 1)), list(range(0, n, 5))]
    return (np.cumsum([0] + [len(r) for r in rows]).astype(np.uint64),
            np.concatenate([np.array(r, dtype=np.int32) for r in rows]))


@pytest.fixture(scope="module")
def ctx():
    c = pm.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [2047, 2048, 4095, 4096, 4097, 8200])
@pytest.mark.parametrize("labels", [0, 2])
def test_long_lists(ctx, n, labels):
    rp, ci = hubs(n)
    lab = (np.arange(n + 3) % max(labels, 1)).astype(np.uint32) if labels else None
    g = pm.GraphPreprocessor.from_host(pm.HostGraph(rp, ci, lab), labeled=labels > 0)
    for k, e in (P.cycle(5), P.house(), P.cycle_tail(4, 1), P.path(5), P.house_tail(1)):
        text = P.to_g(k, e, [i % 2 for i in range(k)] if labels else None)
        p = pm.PatternPreprocessor(text=text, labeled=labels > 0)
        nr = ctx.count_roots(g, p)
        for b, end in ((0, 12), (nr // 2, nr // 2 + 12), (max(0, nr - 6), nr)):  # ring vertices' roots, and hubs'
            out = []
            for leaf, split in ((0, 0), (0, 2), (0, -1), (1, 0)):
                per = torch.zeros(max(1, nr), dtype=torch.int64, device="cuda")
                reads = torch.zeros(max(1, nr), device="cuda")
                torch.cuda.synchronize()
                c, st = ctx.match(g, [p], root_begin=b, root_end=end, leaf_per_lane=leaf, split_level1=split,
                                  root_counts_ptr=per.data_ptr(), root_reads_ptr=reads.data_ptr(), timeout_ms=60000)
                out.append((c[0], st["n_roots"], st["set_ops"], st["alg_bytes"], per.cpu().numpy(), reads.cpu().numpy()))
            want = out[-1]
            for got in out[:-1]:
                assert got[:4] == want[:4], (k, e, b)
                assert np.array_equal(got[4], want[4])
            assert np.array_equal(out[0][5], out[1][5]) and np.array_equal(out[0][5], out[2][5])
    g.close()
