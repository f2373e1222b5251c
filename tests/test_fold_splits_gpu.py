"""Contiguous folds on either side of the limits between 8, 32 and 256 threads a
segment and between one chunk a segment and several; variances of the shortest
segments.  Oracle and tolerances of test_fold_gpu.py, variances within two ulps."""
import numpy as np
import pytest
import torch

from test_fold_gpu import _data, _same_bits, _ulp32

pytestmark = pytest.mark.gpu

SHAPES = [(1, 65, 1215), (1, 65, 1216), (1, 128, 1216), (1, 129, 1216), (1, 256, 4864), (1, 257, 4864), (1, 640, 9728), (1, 641, 9728),
          (1, 640, 9727), (1, 600, 607), (1, 600, 608), (1, 1025, 608), (1, 1025, 1216), (1, 4096, 1823), (1, 4096, 1824),
          (1, 8192, 2431), (1, 8192, 2432), (1, 8191, 3), (1, 8192, 3), (1, 32767, 304), (1, 32768, 304), (1, 20000, 303),
          (1, 131073, 9), (1, 16385, 3000)]
SHORT = [(1, n, 1500) for n in (1, 2, 3, 5, 7, 8, 9, 10, 15, 63, 64)]


@pytest.mark.parametrize("op", ["sum", "max", "stdev"])
@pytest.mark.parametrize("shape", SHAPES + SHORT, ids=lambda s: "x".join(map(str, s)))
def test_threads_and_chunks(lib, dev, oracle, shape, op):
    x = _data(shape, op, 83)
    got = lib.fold(torch.from_numpy(x).to(dev), *shape, op, index=op == "max")
    ref, _, ridx = oracle.fold_ref(x, *shape, op)
    if op == "max":
        assert _same_bits(got[0].cpu().numpy(), ref.astype(np.float32)) and np.array_equal(got[1].cpu().numpy(), ridx)
    else:
        err = np.abs(got.cpu().numpy().astype(np.float64) - ref)
        assert (err <= (2.0 if op == "stdev" else 1.0) * _ulp32(ref) + 1e-30).all()
