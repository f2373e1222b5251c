"""The functions that a compiled kernel evaluates over a thread's lanes, two to
an instruction, against the interpreter, which evaluates one element at a time:
the same bits over the whole range of float (every exponent and sign, subnormals,
infinities, NaN, and the values around each function's limits), with common and
special values side by side in one thread and a partly filled last vector.  The
hand-written form of exp(-x^2) sqrt|y| + log1p|z| takes its four lanes the same
way; shifted by one element it goes one at a time."""
import numpy as np
import pytest
import torch

from nt2_gb300 import expr as E

pytestmark = pytest.mark.gpu

JIT, INTERP = 1, 2

EDGES = np.array([0.0, 1.0, 0.5, 2.0, 4.0, 88.0, 88.3762626647949, 88.72283, 87.33654, 103.0, 104.0, 128.0, 2.0**-24,
                  2.0**-126, 2.0**-149, 2.0**24, 2.0**126, 2.0**127, 3.4028235e38, 0.78539816, 1.5707964, 255.0,
                  10.0, 10.0543, 14.5, 0.70710678, 0.9999999, 1.0000001, 6.5, 13.0, 35.0, np.inf, np.nan], np.float32)


def _sweep(order, rng):
    """4.2 million floats: every 1021st bit pattern, and the edges and their neighbours."""
    bits = (np.arange((1 << 22) - 4096, dtype=np.uint64) * 1021 % (1 << 32)).astype(np.uint32)
    e = np.concatenate([EDGES, -EDGES]).view(np.uint32)
    near = (e[:, None].astype(np.int64) + np.arange(-8, 9)).ravel()
    x = np.concatenate([bits, (near % (1 << 32)).astype(np.uint32)]).view(np.float32)
    if order == "mixed":
        x = rng.permutation(x)
    return x[: x.size - x.size % 4 + 3]


def _same(a, b):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    bad = (a.view(np.uint32) != b.view(np.uint32)) & ~(np.isnan(a) & np.isnan(b))
    assert not bad.any(), (int(bad.sum()), np.flatnonzero(bad)[:4])


@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("name", ["exp", "log", "log1p", "sin", "cos", "erf", "gammaln", "normcdf", "fastnormcdf", "pow"])
def test_lanes_match_one_element_at_a_time(lib, dev, name, order):
    rng = np.random.default_rng(29)
    x = _sweep(order, rng)
    tx = torch.from_numpy(x).to(dev)
    f = getattr(E, name)
    if name == "pow":
        ty = torch.from_numpy(_sweep("mixed", rng)[: x.size].copy()).to(dev)
        tz = torch.from_numpy(rng.uniform(-30, 30, x.size).astype(np.float32)).to(dev)  # most results in range
        exprs = [f(E.Table(tx), E.Table(ty)), f(E.abs_(E.Table(tx)), E.Table(tz))]
    else:
        exprs = [f(E.Table(tx)), f(E.Table(tx)) * E.Table(tx)]
    outs = {m: [torch.full_like(tx, 7.0) for _ in exprs] for m in (JIT, INTERP)}
    for m in (JIT, INTERP):
        prog = E.assign(outs[m], exprs, force_generic=m)
    prog.jit_prepare(0)  # raises if the compiled kernel is unavailable
    for a, b in zip(outs[JIT], outs[INTERP]):
        _same(a, b)


@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("prec", ["fast", "nt2"])
def test_expr3_four_at_a_time_matches_one(lib, dev, prec, order):
    p = lib.PREC_NT2 if prec == "nt2" else lib.PREC_FAST
    rng = np.random.default_rng(31)
    xs = [_sweep(order, rng), _sweep("mixed", rng), np.roll(_sweep(order, rng), 5)]
    n = xs[0].size
    aligned = [torch.from_numpy(a).to(dev) for a in xs]
    shifted = [torch.empty(n + 1, device=dev)[1:].copy_(t) for t in aligned]
    o4, o1 = torch.full((n,), 7.0, device=dev), torch.full((n + 1,), 7.0, device=dev)[1:]
    lib.expr3(*aligned, o4, precision=p)
    lib.expr3(*shifted, o1, precision=p)
    _same(o4, o1)
