"""Folds whose loads run ahead through shared memory, at the edges of a thread's
ring (rows a thread: none, one, a slot less one, whole slots and one more), and
folds of a few long segments either side of the two limits of the one-wave plan
(304 segments, 2^25 elements).  Oracle and tolerances of test_fold_gpu.py."""
import numpy as np
import pytest
import torch

from test_fold_gpu import _data, _same_bits, _ulp32

pytestmark = pytest.mark.gpu

RINGS = [(1, n, 1300) for n in (300, 384, 508, 512, 516, 1020, 1024, 1028, 1152)]      # 32 threads: 128 elements a row
RINGS += [(1, n, 5000) for n in (68, 96, 124, 128, 132, 160, 252)]                      # 8 threads: 32 elements a row
RINGS += [(128, n, 3) for n in (1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 56, 63, 64, 65, 72)]  # a warp every eighth row
WAVES = [(1, 5000, 303), (1, 5000, 304), (1, 5000, 305), (1, 1 << 25, 1), (1, (1 << 25) + 4, 1), (1, 110376, 304),
         (1, 110380, 304)]


@pytest.mark.parametrize("op", ["sum", "max", "stdev"])
@pytest.mark.parametrize("shape", RINGS + WAVES, ids=lambda s: "x".join(map(str, s)))
def test_folds_ahead(lib, dev, oracle, shape, op):
    x = _data(shape, "sum" if op == "stdev" else op, 57)
    t = torch.from_numpy(x).to(dev)
    if op == "max":
        out, idx = lib.fold(t, *shape, op, index=True)
        ref, _, ridx = oracle.fold_ref(x, *shape, op)
        assert _same_bits(out.cpu().numpy(), ref.astype(np.float32)) and np.array_equal(idx.cpu().numpy(), ridx)
        return
    got = lib.fold(t, *shape, op).cpu().numpy().astype(np.float64)
    if op == "sum":
        ref, _, _ = oracle.fold_ref(x, *shape, op)
        assert (np.abs(got - ref) <= _ulp32(ref)).all()
        return
    v = x.astype(np.float64).reshape(shape[2], shape[1], shape[0])
    ref = v.std(axis=1, ddof=1).ravel() if shape[1] > 1 else np.zeros(shape[0] * shape[2])
    assert (np.abs(got - ref) <= 2.0 * _ulp32(np.maximum(ref, 1e-30))).all()
