"""Running sums of long whole segments: as many bits carried from tile to tile as
FP64 holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_running_sum_of_a_long_segment_keeps_fp64(lib, dev):
    """What is left after the large addends cancel again, several tiles on."""
    n, hi = 5 * 16384, 1824
    x = torch.zeros(hi, n, device=dev)
    for k, v in enumerate((1.0, 2.0 ** -25, 2.0 ** -50, -1.0, -2.0 ** -25)):
        x[:, 16384 * k + 5] = v
    got = lib.scan(x.view(-1), 1, n, hi, "sum").view(hi, n)
    assert (got[:, -1] == 2.0 ** -50).all()
