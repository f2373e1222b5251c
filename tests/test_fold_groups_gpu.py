"""The folds' work splits at their edges: 8, 32 or 256 threads a contiguous
segment, chunked segments, several segments a block, segments that start off a
16-byte boundary, strided chunks; the one-pass variance on its difficult data
(a far-off pivot, a large mean, squares past the float range, infinities and
NaN); the extremes' zeros and ties.  The oracle and tolerances are those of
test_fold_gpu.py; variances within 2 ulps of FP64."""
import numpy as np
import pytest
import torch

from test_fold_gpu import _data, _same_bits, _ulp32

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 64, 1024), (1, 65, 5000), (1, 33, 1000), (1, 256, 5001), (1, 257, 5000),   # a thread, 8, 32 threads a segment
    (1, 65, 300), (1, 513, 1215), (1, 513, 1217), (1, 2049, 3647), (1, 2050, 3649),  # 32 or 256 by their number
    (1, 4096, 30), (1, 4097, 30), (1, 12289, 200), (1, 999999, 1), (1, 5, 3),        # chunks
    (33, 63, 1), (32, 64, 1), (128, 640, 3), (131, 641, 3), (4, 100003, 1), (7, 3, 900), (2432 * 128, 5, 1), (2048, 20000, 1), (40, 40000, 1),  # strided
]


@pytest.mark.parametrize("op", ["sum", "max", "min", "asum2", "prod"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_fold_splits(lib, dev, oracle, shape, op):
    x = _data(shape, op, 51)
    idx = op in ("max", "min")
    got = lib.fold(torch.from_numpy(x).to(dev), *shape, op, index=idx)
    ref, _, ridx = oracle.fold_ref(x, *shape, op)
    if idx:
        assert _same_bits(got[0].cpu().numpy(), ref.astype(np.float32))
        assert np.array_equal(got[1].cpu().numpy(), ridx)
        assert _same_bits(lib.fold(torch.from_numpy(x).to(dev), *shape, op).cpu().numpy(), ref.astype(np.float32))
        return
    err = np.abs(got.cpu().numpy().astype(np.float64) - ref)
    assert (err <= (2.0 if op == "prod" else 1.0) * _ulp32(ref)).all()


@pytest.mark.parametrize("off", [1, 2, 3])
@pytest.mark.parametrize("shape", [(1, 40, 2000), (1, 1001, 1300), (1, 300000, 2), (64, 200, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_fold_off_a_boundary(lib, dev, oracle, shape, off):
    x = _data(shape, "max", 52)
    t = torch.zeros(x.size + 4, device=dev)[off:off + x.size]
    t.copy_(torch.from_numpy(x))
    out, idx = lib.fold(t, *shape, "max", index=True)
    ref, _, ridx = oracle.fold_ref(x, *shape, "max")
    assert _same_bits(out.cpu().numpy(), ref.astype(np.float32)) and np.array_equal(idx.cpu().numpy(), ridx)
    ref, _, _ = oracle.fold_ref(x, *shape, "sum")
    err = np.abs(lib.fold(t, *shape, "sum").cpu().numpy().astype(np.float64) - ref)
    assert (err <= _ulp32(ref)).all()


def _var64(x, shape):
    return x.astype(np.longdouble).reshape(shape[2], shape[1], shape[0]).var(axis=1, ddof=1).ravel().astype(np.float64)


@pytest.mark.parametrize("shape", [(1, 16, 1024), (1, 40, 2000), (1, 90, 5000), (1, 1000, 1300), (1, 5000, 20), (1, 300001, 2),
                                   (5, 1000, 2), (64, 3000, 1)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["plain", "mean", "pivot", "ramp", "scales", "constant"])
def test_variance_one_pass(lib, dev, shape, kind):
    lo, n, hi = shape
    rng = np.random.default_rng(53)
    x = rng.standard_normal((hi, n, lo))
    if kind == "mean":
        x += 1000.0
    elif kind == "pivot":  # the first element far from all others
        x[:, 0, :] = 3000.0
    elif kind == "ramp":
        x += np.linspace(-50, 50, n)[None, :, None]
    elif kind == "scales":
        x *= np.exp2(rng.integers(-20, 20, x.shape))
    elif kind == "constant":
        x[:] = 0.1
    x = x.astype(np.float32).ravel()
    ref = _var64(x, shape)
    got = lib.fold(torch.from_numpy(x).to(dev), *shape, "var").cpu().numpy().astype(np.float64)
    assert (np.abs(got - ref) <= 2 * _ulp32(ref)).all()


@pytest.mark.parametrize("shape", [(1, 16, 1024), (1, 48, 1000), (1, 5000, 4), (1, 300001, 1), (8, 1000, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_variance_at_the_float_range(lib, dev, shape):
    """Deviations whose squares fit, from a pivot whose squares do not; an
    infinity or a NaN among the elements gives 0, as in the two-pass form."""
    lo, n, hi = shape
    rng = np.random.default_rng(54)
    x = rng.uniform(-1, 1, (hi, n, lo)) * 1e16
    x[:, 0, :] = 1.8e19  # its square about the mean is 3.2e38; n squares of the others about it are past 3.4e38
    x = x.astype(np.float32)
    ref = _var64(x.ravel(), shape)
    got = lib.fold(torch.from_numpy(x.ravel()).to(dev), *shape, "var").cpu().numpy().astype(np.float64)
    assert (np.abs(got - ref) <= 2 * _ulp32(ref)).all()
    for bad in (np.inf, -np.inf, np.nan):
        y = np.ones((hi, n, lo), np.float32)
        y[:, n // 2, :] = bad
        assert (lib.fold(torch.from_numpy(y.ravel()).to(dev), *shape, "var").cpu().numpy() == 0).all()
