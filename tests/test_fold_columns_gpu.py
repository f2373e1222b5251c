"""Strided folds a thread per output: row counts and outputs on either side of the
limits between that and a block's warps, tables on and off a 16-byte boundary,
and an expression's elements.  Oracle and tolerances of test_fold_gpu.py;
variances within two ulps."""
import numpy as np
import pytest
import torch

from nt2_gb300 import expr as E
from test_fold_gpu import _data, _same_bits, _ulp32

pytestmark = pytest.mark.gpu

SHAPES = [(4, 1, 5), (3, 1, 5), (64, 2, 3), (31, 3, 7), (128, 5, 3), (9, 7, 11), (8, 8, 1), (8, 9, 1), (5, 8, 4), (5, 9, 4),
          (16384, 20, 1), (16384, 21, 1), (65536, 31, 1), (65536, 32, 1), (16385, 31, 1), (16385, 32, 1), (333, 10, 50),
          (49153, 48, 1), (155649, 33, 1), (622592, 33, 1)]


def _check(got, x, shape, op, oracle):
    if op == "max":
        ref, _, ridx = oracle.fold_ref(x, *shape, op)
        assert _same_bits(got[0].cpu().numpy(), ref.astype(np.float32)) and np.array_equal(got[1].cpu().numpy(), ridx)
        return
    got = got.cpu().numpy().astype(np.float64)
    ref, _, _ = oracle.fold_ref(x, *shape, op)
    tol = {"stdev": 2.0, "meanad": 2.0, "prod": 2.0}.get(op, 1.0)
    assert (np.abs(got - ref) <= tol * _ulp32(ref) + 1e-30).all()


@pytest.mark.parametrize("op", ["sum", "max", "stdev", "mean", "prod", "norm2", "meanad", "nbtrue"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_thread_per_output(lib, dev, oracle, shape, op):
    x = _data(shape, op, 81)
    t = torch.from_numpy(x).to(dev)
    _check(lib.fold(t, *shape, op, index=op == "max"), x, shape, op, oracle)
    off = torch.empty(x.size + 1, device=dev)[1:]
    off.copy_(t)
    _check(lib.fold(off, *shape, op, index=op == "max"), x, shape, op, oracle)
    _check(E.fold(E.Table(t) * 1.0, op, shape=shape, index=op == "max"), x, shape, op, oracle)
    if op == "sum":  # the FP64 result, and the float rounded from the same pair
        out, out64 = E.fold(E.Table(t) * 1.0, op, shape=shape, out64=True)
        ref, asum, _ = oracle.fold_ref(x, *shape, op)
        assert (np.abs(out64.cpu().numpy() - ref) <= 4 * 2.0 ** -48 * asum).all()
