"""Strided scans: the last rows in groups of eight, four and one, fewer columns than
a block has threads, and chunks on either side of the limits up to which the scan
adds up their prefixes itself (7 with four columns a thread and for the maxima of
few, 64 else).  Oracle and tolerances of test_scan_tiles_gpu.py."""
import pytest
import torch

from test_scan_gpu import _data
from test_scan_tiles_gpu import _check

pytestmark = pytest.mark.gpu

SHAPES = [(33, n, 2) for n in (1, 3, 4, 7, 8, 9, 12, 15, 16, 17, 23, 31)] + [(36, n, 2) for n in (1, 3, 4, 5, 8, 11, 12, 13)]
SHAPES += [(2, 111, 1), (2, 112, 1), (2, 128, 1), (31, 127, 1), (31, 128, 1), (4, 112, 1), (4, 127, 1), (4, 128, 1), (1024, 127, 1),
           (1024, 128, 1), (1023, 127, 1), (1023, 128, 1), (1025, 127, 1), (1025, 128, 1), (1023, 1040, 1), (1025, 1040, 1),
           (255, 300, 1), (257, 300, 1), (3, 16 * 64, 1), (3, 16 * 66, 1)]


@pytest.mark.parametrize("op", ["sum", "prod", "max", "min"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_strided(lib, dev, oracle, shape, op):
    x = _data(shape, op, 93, nan=True)
    t = torch.from_numpy(x).to(dev)
    _check(lib.scan(t, *shape, op).cpu().numpy(), x, shape, op, oracle)
    lib.scan(t, *shape, op, out=t)  # in place
    _check(t.cpu().numpy(), x, shape, op, oracle)
