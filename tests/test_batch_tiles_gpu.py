"""A batch's default tile: one to eight float4 vectors a thread by the batch's
total size, the same results as with a stated tile."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [1, 127, 5000, 7_000_000, 40_000_000], ids=str)
def test_default_tiles_match_stated_ones(lib, dev, total):
    rng = np.random.default_rng(37)
    cuts = np.unique(rng.integers(0, total + 1, 6)) if total > 100 else np.array([], np.int64)
    sizes = [int(s) for s in np.diff(np.concatenate([[0], cuts, [total]])) if s > 0]
    big = [torch.rand(n, device=dev) * 25 + 5 for n in sizes]
    big2 = [torch.rand(n, device=dev) * 9 + 0.25 for n in sizes]
    L, res = lib.load(), []
    for tune in (None, lib.BatchTune(256, 0, 4, lib.PREC_FAST, 1), lib.BatchTune(0, 0, 0, lib.PREC_FAST, 0)):
        outs = [[torch.zeros(n, device=dev), torch.zeros(n, device=dev)] for n in sizes]
        items = (lib.BatchItem * len(sizes))()
        for i, n in enumerate(sizes):
            items[i].expr, items[i].n = (lib.BATCH_BLACKSCHOLES, lib.BATCH_EXPR3)[i % 2], n
            items[i].inp[0], items[i].inp[1], items[i].inp[2] = (t[i].data_ptr() for t in (big, big, big2))
            items[i].out[0], items[i].out[1] = outs[i][0].data_ptr(), outs[i][1].data_ptr()
            items[i].s[0], items[i].s[1] = 0.3, 0.02
        h = ctypes.c_void_p()
        lib.check(L.nt2g_batch_create(items, len(sizes), ctypes.byref(tune) if tune else None, ctypes.byref(h)))
        try:
            lib.check(L.nt2g_batch_run(h, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            torch.cuda.synchronize()
        finally:
            L.nt2g_batch_destroy(h)
        res.append(outs)
    for other in res[1:]:
        for a, b in zip(res[0], other):
            assert all(torch.equal(u, v) for u, v in zip(a, b))
    assert all(bool(torch.isfinite(o[0]).all()) for o in res[0])
