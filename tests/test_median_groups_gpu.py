"""Medians of strided slices on either side of the limits between eight, four and
one slice a block (76 and 25 blocks).  Equal to a sort."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(600, 1100, 1), (601, 1101, 1), (8, 1030, 75), (8, 1031, 76), (96, 1100, 1), (97, 1100, 1), (100, 9000, 1), (101, 9001, 1),
          (4, 1500, 24), (4, 1500, 25), (7, 2000, 40)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_slices_a_block(lib, dev, shape):
    lo, n, hi = shape
    rng = np.random.default_rng(95)
    x = rng.standard_normal((hi, n, lo)).astype(np.float32)
    x[:, : n // 3] = rng.integers(-3, 4, (hi, n // 3, lo))
    v = np.sort(x, axis=1)
    a, b = v[:, (n - 1) // 2], v[:, n // 2]
    ref = (a + (b - a) * np.float32(0.5)).astype(np.float32) if n % 2 == 0 else a
    got = lib.median(torch.from_numpy(x.ravel()).to(dev), *shape).cpu().numpy()
    assert np.array_equal(got, ref.ravel())
