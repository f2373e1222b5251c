"""Running products through the conversion by bits: plain factors, a zero, a
subnormal factor that a large one makes up for, infinities and NaN, in packed
short segments, segments around a tile's and a run's end, chunked ones and
strided ones of one and four columns a thread; within two ulps of FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 17, 963), (1, 17, 5000), (1, 1000, 50), (1, 1152, 3), (1, 1153, 3), (1, 2177, 2), (1, 4224, 2), (1, 4225, 3), (1, 5000, 7),
          (1, 40000, 2), (40, 300, 2), (33, 300, 2), (64, 5000, 1)]


@pytest.mark.parametrize("kind", ["plain", "zero", "subnormal", "inf", "nan"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_products(lib, dev, shape, kind):
    lo, n, hi = shape
    rng = np.random.default_rng(91)
    x = (rng.uniform(0.999, 1.001, (hi, n, lo)) * rng.choice([-1.0, 1.0], (hi, n, lo))).astype(np.float32)
    at = n * 2 // 3
    if kind == "subnormal":  # down to 2^-143 and back to 2^-16
        x[:, at - 5] = np.float32(2.0 ** -143) * 1.0
        x[:, at] = np.float32(2.0 ** 127)
    elif kind != "plain":
        x[:, at] = {"zero": -0.0, "inf": np.inf, "nan": np.nan}[kind]
    ref = np.cumprod(x.astype(np.float64), axis=1).ravel()
    got = lib.scan(torch.from_numpy(x.ravel()).to(dev), *shape, "prod").cpu().numpy()
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    r32 = ref.astype(np.float32)
    big = np.isinf(r32) | (r32 == 0.0)
    assert np.array_equal(got[big & ~nan].view(np.uint32), r32[big & ~nan].view(np.uint32))
    ok = ~nan & ~big
    assert (np.abs(got[ok].astype(np.float64) - ref[ok]) <= 2 * np.spacing(np.abs(r32[ok])).astype(np.float64)).all()
