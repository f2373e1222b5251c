"""Reverse mode where a thread's next elements wait in shared memory: sizes
around a pair, a block's tile, one and two waves of blocks; up to eight tables
(cotangents included), more than that (direct loads), a uint8 table among them,
a missing cotangent.  The same bits as the same tables one element off a 16-byte
boundary, which go element by element; scalars' sums agree to the rounding of
compensated float sums."""
import numpy as np
import pytest
import torch

from nt2_gb300 import expr as E

pytestmark = pytest.mark.gpu

N = [1, 2, 3, 255, 511, 512, 513, 4097, 152 * 4 * 512, 152 * 8 * 512 + 1, 3_735_551, 5_500_003]


def _pair(dev, n, kind):
    """The table at a 16-byte boundary and a copy one element after one."""
    g = torch.Generator(device=dev)
    g.manual_seed(n % 1000 + len(kind))
    if kind == "byte":
        a = torch.randint(0, 2, (n,), device=dev, generator=g, dtype=torch.uint8)
    else:
        a = torch.rand(n, device=dev, generator=g) * (1.5 if kind == "ct" else 20.0) + 0.25
    b = torch.empty(n + 1, device=dev, dtype=a.dtype)[1:]
    b.copy_(a)
    return a, b


@pytest.mark.parametrize("form", ["ring", "direct", "byte"])
@pytest.mark.parametrize("n", N)
def test_reverse_mode_ahead_matches_element_by_element(lib, dev, n, form):
    tables = 9 if form == "direct" else 3
    pairs = [_pair(dev, n, "in" * (k + 1)) for k in range(tables)]
    byte = _pair(dev, n, "byte")
    cts = [_pair(dev, n, "ct" + "t" * k) for k in range(2)]
    res = []
    for side in (0, 1):
        t = [p[side] for p in pairs]
        T = [E.Table(x) for x in t]
        r = E.Scalar(0.02)
        e1 = E.log(T[0] / T[1]) * E.exp(-r * T[2]) + E.normcdf(T[0] - T[1])
        e2 = E.sqrt(T[0] * T[2]) - T[1] * r
        for x in T[3:]:
            e1 = e1 * x + E.sqr(x)
        if form == "byte":
            e2 = E.if_else(E.Table(byte[side]) > E.Scalar(0, lib.U8), e2, T[1])
        outs = [torch.empty_like(t[0]) for _ in range(2)]
        for ct in ([c[side] for c in cts], [cts[0][side], None]):
            res.append((side, E.vjp(outs, [e1, e2], ct, t + [r])))
    torch.cuda.synchronize()
    for (_, a), (_, b) in zip(res[:2], res[2:]):
        for u, v in zip(a[:-1], b[:-1]):
            assert torch.equal(u.view(torch.int32), v.view(torch.int32))
        # every addend within 2^-46 of its sum's magnitude: log, exp and the cotangents stay below 100
        assert abs(float(a[-1]) - float(b[-1])) <= 2.0 ** -44 * n * 100.0


@pytest.mark.parametrize("n", [1, 2, 513, 300_001])
def test_scalar_gradient_of_extreme_adjoints(lib, dev, n):
    """A scalar's gradient in FP64 range: adjoints past 2^96 whose float sum would
    overflow, huge ones that cancel, infinities and NaN."""
    x = np.full(n, 1.0, np.float32)
    for big in (np.float32(3e38), np.float32(2.0 ** 96), np.float32(-1e30)):
        t, ct = torch.from_numpy(x).to(dev), torch.full((n,), float(big), device=dev)
        if n > 2:
            ct[1::2] = -float(big)
            ct[0] = 1.0
        r = E.Scalar(0.5)
        (g,) = E.vjp([torch.empty_like(t)], [E.Table(t) * r], [ct], [r])
        want = ct.double().sum().item()
        assert abs(float(g) - want) <= 2.0 ** -50 * float(ct.double().abs().sum())
    ct = torch.ones(n, device=dev)
    for v in (float("inf"), float("-inf"), float("nan")):
        ct[n // 2] = v
        r = E.Scalar(0.5)
        (g,) = E.vjp([torch.empty_like(t)], [E.Table(t) * r], [ct], [r])
        assert (np.isnan(float(g)) if np.isnan(v) else float(g) == v)
