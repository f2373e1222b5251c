"""The lanes' reciprocal (one Newton step on the approximate one) inside the
functions that use it, over all 2^23 significands of its operand: the bits of
the interpreter, which divides."""
import numpy as np
import pytest
import torch

from nt2_gb300 import expr as E

pytestmark = pytest.mark.gpu

SIGNIFICANDS = np.arange(1 << 23, dtype=np.uint32)


# the operand: x itself from 6.5 on; 1 + x; the significand in [sqrt(1/2), sqrt(2)), plus 1
CASES = {"gammaln": (E.gammaln, 8.0), "log1p": (E.log1p, None), "pow": (lambda x: E.pow(x, E.Scalar(1.7)), 1.0)}


@pytest.mark.parametrize("name", CASES)
def test_every_significand(lib, dev, name):
    f, base = CASES[name]
    x = ((np.float32(2.0 if base is None else base).view(np.uint32) + SIGNIFICANDS).view(np.float32))
    if base is None:
        x = (x.astype(np.float64) - 1.0).astype(np.float32)  # 1 + x takes every value of [2, 4)
        assert np.array_equal((np.float32(1) + x).view(np.uint32) & 0x7fffff, SIGNIFICANDS)
    t = torch.from_numpy(x).to(dev)
    outs = [torch.full_like(t, 7.0) for _ in range(2)]
    for mode, o in zip((1, 2), outs):
        E.assign([o], [f(E.Table(t))], force_generic=mode)
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))
