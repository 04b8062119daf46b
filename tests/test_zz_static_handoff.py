"""Work hand-off in the allocation-free entry, whose ring has fewer slots than warps may wait: several waiting warps
share a slot, and no piece is lost or torn.  (Collected last, like the entry's other tests.)"""
import ctypes as C

import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("occupancy", [1, 2])
@pytest.mark.parametrize("shape", [P.cycle(6), P.house_tail(1)])
def test_more_waiting_warps_than_slots(shape, occupancy):
    n = 40  # a complete graph: few roots, each a search of its own size
    rp = (np.arange(n + 1) * (n - 1)).astype(np.uint64)
    ci = np.concatenate([[j for j in range(n) if j != i] for i in range(n)]).astype(np.int32)
    d_rp, d_ci = torch.from_numpy(rp.astype(np.int64)).cuda(), torch.from_numpy(ci).cuda()
    p = pm.PatternPreprocessor(text=P.to_g(*shape), labeled=False)
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(pm.HostGraph(rp, ci))
    want, wst = ctx.match(g, [p], timeout_ms=60000)
    o = pm.Context._opts(high_occupancy=occupancy, split_level1=2, timeout_ms=60000)
    for _ in range(3):
        cnt, st = C.c_uint64(), pm.Stats()
        rc = pm.lib().pm_match_static(C.c_void_p(d_rp.data_ptr()), C.c_void_p(d_ci.data_ptr()), None, n, len(ci), n - 1,
                                      p._h, C.byref(o), None, C.byref(cnt), C.byref(st))
        assert rc == pm.PM_OK, pm.lib().pm_last_error()
        st = st.as_dict()
        assert st["grid_blocks"] * st["block_threads"] // 32 > 8 * 256  # warps past the ring's slots
        assert st["splits"] > 1000
        assert (cnt.value, st["set_ops"], st["alg_bytes"]) == (want[0], wst["set_ops"], wst["alg_bytes"])
    g.close()
    ctx.close()
