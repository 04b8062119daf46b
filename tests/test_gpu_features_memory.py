"""Root features with no room for a row per vertex: each root by itself, as good."""
import ctypes as C

import numpy as np
import pytest
import torch

import pumatch_b200 as pm
from pumatch_b200 import learn
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def test_features_without_room_for_rows():
    n = 4_000_000  # 256 MB of rows
    v = np.arange(n, dtype=np.int64)
    ci = np.sort(np.stack([(v - 1) % n, (v + 1) % n], axis=1), axis=1).astype(np.int32).ravel()
    labels = (v % 1000 == 0).astype(np.uint32)  # label 1 on every thousandth vertex of a ring
    hg = pm.HostGraph(np.arange(0, 2 * n + 1, 2, dtype=np.uint64), ci, labels)
    g = pm.GraphPreprocessor.from_host(hg, labeled=True)
    p = pm.PatternPreprocessor(text=P.to_g(*P.path(4), [1, 0, 0, 0]), labeled=True)
    roomy, tight = pm.Context(0), pm.Context(0)
    want = learn.root_features(roomy, g, p)
    gu = pm.GraphPreprocessor.from_host(pm.gen_chung_lu(400, 2000, seed=1))  # the kernel for single roots, loaded
    learn.root_features(tight, gu, pm.PatternPreprocessor(text=P.to_g(*P.path(4)), labeled=False))
    assert len(tight.roots(g, p)) == want.shape[0] > 0
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    hold, size = [], 1 << 33
    while size >= 1 << 25:  # all but some tens of megabytes of the device
        try:
            hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size >>= 1
    try:
        assert torch.cuda.mem_get_info()[0] < n * 64
        got = C.c_int64()
        rc = pm.lib().pm_root_features(tight._h, g._h, p._h, C.c_void_p(out.data_ptr()), out.shape[0], C.byref(got))
        assert rc == pm.PM_OK, pm.lib().pm_last_error()
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert got.value == want.shape[0]
    torch.testing.assert_close(out, want, rtol=1e-5, atol=1e-5)
    for x in (g, gu, roomy, tight):
        x.close()
