"""Maxima and minima of data that hold the fold's neutral value (-inf for max,
+inf for min: log-probabilities, masked elements) or its opposite: slices of
nothing else, one number among them, infinities only at a slice's ends, in a
few of its rows or in one half of it, and beside a NaN; values and positions
against the oracle, on every route of a fold (a thread, 8, 32 or 256 threads a
segment, chunks, strided rows one or four to a load), from tables on and off a
16-byte boundary and from expressions."""
import numpy as np
import pytest
import torch

from nt2_gb300 import expr as E
from test_fold_gpu import _same_bits

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 64, 1024), (1, 68, 5000), (1, 65, 5000), (1, 260, 400), (1, 515, 30), (1, 1024, 8), (1, 2050, 3650),  # a thread, 8, 32 or 256 a segment
    (1, 4096, 3), (1, 5003, 1), (1, 70001, 2), (1, 1 << 20, 1),                                               # chunks
    (5, 8, 3), (7, 24, 2), (31, 25, 1), (9, 1003, 2), (2049, 200, 1), (64, 8, 3), (128, 33, 2), (64, 5000, 1),  # strided
    (300004, 9, 1),
]
KINDS = ["all", "one_number", "ends", "first_half", "every_eighth_row", "last_row", "with_nan", "opposite"]


def _fill(shape, kind, op, seed):
    lo, n, hi = shape
    rng = np.random.default_rng(seed)
    worst = -np.inf if op == "max" else np.inf
    # numbers that a 0 would beat
    x = (rng.uniform(1, 9, (hi, n, lo)) * (-1 if op == "max" else 1)).astype(np.float32)
    if kind == "all":
        x[:] = worst
    elif kind == "one_number":
        keep = rng.integers(0, n, (hi, 1, lo))
        x = np.where(np.arange(n)[None, :, None] == keep, x, np.float32(worst))
    elif kind == "ends":
        x[:, :3] = worst
        x[:, -5:] = worst
    elif kind == "first_half":
        x[:, : (n + 1) // 2] = worst
    elif kind == "every_eighth_row":
        x[:, ::8] = worst
    elif kind == "last_row":
        x[:, -1] = worst
    elif kind == "with_nan":
        x[:] = worst
        x[:, n // 3] = np.nan
    else:
        x[:, n // 2] = -worst
        x[:, -1] = -worst
    return np.ascontiguousarray(x).ravel()


def _check(got, oracle, x, shape, op):
    ref, _, ridx = oracle.fold_ref(x, *shape, op)
    out, idx = got
    assert _same_bits(out.cpu().numpy(), ref.astype(np.float32))
    assert np.array_equal(idx.cpu().numpy(), ridx)


@pytest.mark.parametrize("op", ["max", "min"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_extremes_with_infinities(lib, dev, oracle, shape, kind, op):
    x = _fill(shape, kind, op, 61)
    t = torch.from_numpy(x).to(dev)
    off = torch.empty(x.size + 1, device=dev)[1:]
    off.copy_(t)
    _check(lib.fold(t, *shape, op, index=True), oracle, x, shape, op)
    _check(lib.fold(off, *shape, op, index=True), oracle, x, shape, op)
    plain = lib.fold(t, *shape, op)
    assert _same_bits(plain.cpu().numpy(), lib.fold(t, *shape, op, index=True)[0].cpu().numpy())
    # as an expression's: one table a load, and one off a boundary
    _check(E.fold(E.Table(t) * 1.0, op, shape=shape, index=True), oracle, x, shape, op)
    _check(E.fold(E.Table(off) * 1.0, op, shape=shape, index=True), oracle, x, shape, op)
    assert _same_bits(E.fold(E.Table(t) * 1.0, op, shape=shape).cpu().numpy(), plain.cpu().numpy())
