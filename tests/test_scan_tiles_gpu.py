"""The scan's tiles and chunks at their edges: packed short segments, segments
around one tile (128 threads of 9, 17 or 33 elements), segments of several
chunks, strided chunks whose prefix the scan adds up itself (up to 64) and
more, tables that start off a 16-byte boundary, and the least workspace a call
may pass.  The oracle and tolerances are those of test_scan_gpu.py."""
import numpy as np
import pytest
import torch

from test_scan_gpu import _data, _same_bits

pytestmark = pytest.mark.gpu

TILE = 4224
SHAPES = [
    (1, 1, 1000), (1, 2, 5001), (1, 31, 30000), (1, 1023, 9000), (1, 1023, 9),   # packed
    (1, 1024, 9), (1, 1152, 3), (1, 1153, 3), (1, 2176, 5), (1, 2177, 5),        # a block each, of each run length
    (1, TILE - 1, 5), (1, TILE, 3), (1, TILE + 1, 3),                            # around one tile
    (1, 64 * TILE, 1), (1, 64 * TILE + 1, 1), (1, 1300 * TILE + 7, 2),           # chunks of a tile, of several
    (1, 9001, 5000),                                                             # long segments, a block each
    (31, 4097, 1), (32, 256, 3), (64, 129, 2), (65, 127, 1),                     # strided chunks
    (3000, 900, 1), (2404, 16 * 64, 1), (301, 16 * 128 + 5, 1), (2, 70000, 1),   # around 64 of them
]


def _check(got, x, shape, op, oracle):
    if op in ("max", "min"):
        assert _same_bits(got, oracle.scan_nt2(x, *shape, op))
        return
    if op == "sum":
        ref, absrun = oracle.cumsum_exact(x, *shape)
        tol = np.spacing(np.abs(ref).astype(np.float32)).astype(np.float64) + 1e-12 * absrun
    else:
        ref = np.cumprod(x.astype(np.float64).reshape(shape[2], shape[1], shape[0]), axis=1).ravel()
        tol = 2 * np.spacing(np.abs(ref).astype(np.float32)).astype(np.float64)
    assert (np.abs(got.astype(np.float64) - ref) <= tol).all(), (op, shape)


@pytest.mark.parametrize("op", ["sum", "prod", "max"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_scan_tile_edges(lib, dev, oracle, shape, op):
    x = _data(shape, op, 41, nan=True)
    got = lib.scan(torch.from_numpy(x).to(dev), *shape, op)
    again = lib.scan(torch.from_numpy(x).to(dev), *shape, op)
    assert torch.equal(got.view(torch.int32), again.view(torch.int32))  # a fixed combine order
    _check(got.cpu().numpy(), x, shape, op, oracle)


@pytest.mark.parametrize("op", ["sum", "max"])
@pytest.mark.parametrize("shape", [(1, 3001, 50), (1, TILE + 3, 2), (1, 20 * TILE + 1, 1), (40, 300, 2)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("x_off,out_off", [(1, 1), (3, 0), (0, 2)])
def test_scan_misaligned_and_in_place(lib, dev, oracle, shape, op, x_off, out_off):
    x = _data(shape, op, 42)
    n = x.size
    xs = torch.zeros(n + 8, device=dev)[x_off:x_off + n]
    xs.copy_(torch.from_numpy(x))
    room = torch.full((n + 8,), 7.0, device=dev)
    lib.scan(xs, *shape, op, out=room[out_off:out_off + n])
    got = room.cpu().numpy()
    _check(got[out_off:out_off + n], x, shape, op, oracle)
    assert (got[:out_off] == 7).all() and (got[out_off + n:] == 7).all()
    lib.scan(xs, *shape, op, out=xs)
    assert _same_bits(xs.cpu().numpy(), got[out_off:out_off + n])


def _least_bytes(lo, inner, hi):
    """16 bytes per chunk of the smallest split that occupies the GPU: what a scan has always accepted."""
    def chunks(vec):
        if lo == 1:
            chunk = 16384
            if hi * -(-inner // chunk) < 4864:
                chunk = max(1024, -(-inner // -(-4864 // hi)))
            return -(-inner // (-(-chunk // 512) * 512))
        threads, q = lo * hi // vec, 1
        if threads < 155648:
            q = min(-(-155648 // threads), max(inner // 16, 1), 65535)
        return -(-inner // -(-inner // q))
    q = max(chunks(1), chunks(4) if lo % 4 == 0 else 1)
    return lo * hi * q * 16 if q > 1 else 0


@pytest.mark.parametrize("shape", [(60000, 2000, 1), (1, 50000, 40), (64, 1000, 1)], ids=lambda s: "x".join(map(str, s)))
def test_scan_least_workspace(lib, dev, oracle, shape):
    """A call with that much workspace is accepted, one byte less refused."""
    x = _data(shape, "max", 43)
    xs, least = torch.from_numpy(x).to(dev), _least_bytes(*shape)
    out, ws = torch.empty_like(xs), torch.empty(least, dtype=torch.uint8, device=dev)
    call = lambda b: lib.load().nt2g_scan_f32(lib._ptr(xs), *shape, lib.SCAN["max"], lib.PREC_FAST, lib._ptr(ws), b,  # noqa: E731
                                              lib._ptr(out), lib._stream())
    assert call(least - 1) == lib.ERR_INVALID
    lib.check(call(least))
    assert _same_bits(out.cpu().numpy(), oracle.scan_nt2(x, *shape, "max"))
