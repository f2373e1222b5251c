"""Sums, means and norms whose shares leave the float range though the result
does not, and the bits an FP64 combination of the warps' shares keeps: a
block's warps, its chunks and long whole segments, contiguous and strided; the
bits of a variance whose first element is far from all others."""
import pytest
import torch

from nt2_gb300 import expr as E

pytestmark = pytest.mark.gpu


# (shape, value): no 512 elements of a thread reach 3.4e38, a block's do
MEANS = [((1, 1 << 24, 1), 5e34), ((1, 1000000, 1), 1.5e35), ((1, 4096, 40), 2.5e35), ((1, 3000, 2000), 2.5e35), ((1, 3000, 4000), 2e35), ((1, 200, 6000), 1.5e36), ((1, 200000, 1900), 1.5e34),
         ((1, 40000, 4000), 1.5e34), ((64, 1 << 16, 1), 1e37), ((63, 5000, 2), 1e37), ((300000, 40, 1), 1e37), ((6000, 8192, 1), 2e36)]


@pytest.mark.parametrize("shape,value", MEANS, ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else str(s))
def test_means_of_large_values(lib, dev, shape, value):
    lo, n, hi = shape
    g = torch.Generator(device=dev)
    g.manual_seed(71)
    x = (torch.rand(lo * n * hi, device=dev, generator=g) * 0.25 + 0.75) * value
    exact = (x.view(hi, n, lo).sum(dim=1, dtype=torch.float64) / n).ravel()
    got = lib.fold(x, *shape, "mean").double()
    # half an ulp of the float, and the two FP64 sums' rounding
    assert ((got - exact).abs() <= exact * (2.0 ** -24 + n * 2.0 ** -53)).all()
    _, got64 = E.fold(E.Table(x) * 1.0, "mean", shape=shape, out64=True)
    assert ((got64 - exact).abs() <= exact * (n * 2.0 ** -53 + 2.0 ** -44)).all()


@pytest.mark.parametrize("shape,value", [((1, 1 << 24, 1), 2e17), ((1, 1000000, 1), 4e17), ((6000, 400, 1), 2e18)],
                         ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else str(s))
def test_norms_of_large_values(lib, dev, shape, value):
    lo, n, hi = shape
    g = torch.Generator(device=dev)
    g.manual_seed(72)
    x = (torch.rand(lo * n * hi, device=dev, generator=g) * 0.25 + 0.75) * value
    exact = x.double().square().view(hi, n, lo).sum(dim=1).sqrt().ravel()
    got = lib.fold(x, *shape, "norm2").double()
    assert ((got - exact).abs() <= exact * (2.0 ** -24 + n * 2.0 ** -53)).all()


# a sum that FP64 holds and a pair of floats does not: 1 + 2^-25 + 2^-50
@pytest.mark.parametrize("at", [(0, 1024 + 128, 2048 + 256), (3000, 1030, 5), (40, 77, 4000)], ids=str)
def test_warps_meet_in_fp64(lib, dev, at):
    x = torch.zeros(4096, device=dev)
    for k, v in zip(at, (1.0, 2.0 ** -25, 2.0 ** -50)):
        x[k] = v
    _, total = E.fold(E.Table(x) * 1.0, "sum", out64=True)
    assert total.item() == 1.0 + 2.0 ** -25 + 2.0 ** -50
    rows = x.view(1, 4096).repeat(96, 1).t().contiguous()  # 4096 rows of 96: a strided fold's
    _, total = E.fold(E.Table(rows.reshape(-1)) * 1.0, "sum", shape=(96, 4096, 1), out64=True)
    assert (total == 1.0 + 2.0 ** -25 + 2.0 ** -50).all()


@pytest.mark.parametrize("shape", [(1, 1 << 24, 1), (1, 1 << 17, 300), (1, 20000, 2000), (64, 100000, 1), (1, 60, 5000), (70, 31, 40)],
                         ids=lambda s: "x".join(map(str, s)))
def test_variance_about_a_far_first_element(lib, dev, shape):
    """The first element of every slice far from all others: the squares about it
    would cancel by up to the slice's length.  512 elements a thread in pairs of
    floats (2^-39), a factor of nine at most in cancelling."""
    lo, n, hi = shape
    g = torch.Generator(device=dev)
    g.manual_seed(73)
    x = torch.randn(hi, n, lo, device=dev, generator=g)
    x[:, 0] = 1e4 + torch.rand(hi, lo, device=dev, generator=g)
    d = x.double() - x.double().mean(dim=1, keepdim=True)
    exact = (((d * d).sum(dim=1) - d.sum(dim=1) ** 2 / n) / (n - 1)).ravel()
    _, got = E.fold(E.Table(x.view(-1)) * 1.0, "var", shape=shape, out64=True)
    assert ((got - exact).abs() <= 2.0 ** -35 * exact).all()
