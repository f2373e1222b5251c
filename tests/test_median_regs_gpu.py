"""Medians with the slice's keys in registers: lengths around the short kernel
(1024), each number of keys a thread (16, 32, 40) and of slices a block (8, 4,
1), slices left over by a group, one to four digits (few keys sharing a digit,
most of them, all of them), long slices whose last keys are gathered or all
equal.  Equal to the oracle's sorted middle."""
import numpy as np
import pytest
import torch

from test_median_gpu import _eq

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 1024, 3), (1, 1025, 3), (1, 4096, 2), (1, 4097, 2), (1, 12289, 2), (1, 16384, 1), (1, 16385, 1), (1, 32769, 1),
    (1, 40960, 1), (8, 1025, 2), (9, 1030, 1), (17, 2048, 1), (8, 4097, 1), (11, 5120, 1), (8, 5121, 1), (6, 8193, 1),
    (4, 10240, 2), (5, 10241, 1), (3, 20001, 1), (1, 40961, 2), (1, 250000, 2), (2, 60001, 2),
]


def _keys(kind, n, rng):
    if kind == "normal":
        return rng.standard_normal(n)
    if kind == "uniform":  # a sixth of the keys and more share the first digit
        return rng.uniform(5, 30, n)
    if kind == "near":  # only the last digits differ
        return (np.float32(1.0).view(np.uint32) + rng.integers(0, 5000, n).astype(np.uint32)).view(np.float32)
    if kind == "equal":
        return np.full(n, -2.5)
    x = np.full(n, 1.0)  # two: the middle pair of an even length straddles far values
    x[: n // 2] = -1e30
    return rng.permutation(x)


@pytest.mark.parametrize("kind", ["normal", "uniform", "near", "equal", "two"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_median_of_keys_in_registers(lib, dev, oracle, shape, kind):
    rng = np.random.default_rng(61)
    x = _keys(kind, shape[0] * shape[1] * shape[2], rng).astype(np.float32)
    if kind == "two":  # each slice its own half and half
        x = np.stack([_keys(kind, shape[1], rng) for _ in range(shape[0] * shape[2])]).astype(np.float32)
        x = x.reshape(shape[2], shape[0], shape[1]).transpose(0, 2, 1).copy().ravel()
    t = torch.from_numpy(x).to(dev)
    for op in ("median", "medianad"):
        assert _eq(lib.median(t, *shape, op).cpu().numpy(), oracle.median(x, *shape, ad=op == "medianad")), op


@pytest.mark.parametrize("shape", [(1, 3001, 4), (9, 3000, 1), (1, 100000, 2)], ids=lambda s: "x".join(map(str, s)))
def test_median_infinities_and_nan(lib, dev, oracle, shape):
    rng = np.random.default_rng(62)
    lo, n, hi = shape
    x = rng.standard_normal((hi, n, lo)).astype(np.float32)
    x[:, rng.permutation(n)[: n // 2 + 2], :] = np.inf  # the middle is +inf: the padding's own key
    y = -x
    z = x.copy()
    z[0, n // 3, 0] = np.nan
    for a in (x, y, z):
        a = a.ravel()
        got = lib.median(torch.from_numpy(a).to(dev), lo, n, hi).cpu().numpy()
        ref = oracle.median(np.nan_to_num(a, nan=0.0, posinf=np.inf, neginf=-np.inf), lo, n, hi)
        if np.isnan(a).any():
            assert np.isnan(got[0]) and _eq(got[1:], ref[1:])
        else:
            assert _eq(got, ref)
