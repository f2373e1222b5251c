"""Inputs of reverse mode that are no argument of the program: a table it does
not read, another Scalar, a plain number."""
import pytest
import torch

from nt2_gb300 import expr as E


def test_what_is_no_argument():
    t, r = torch.zeros(4), E.Scalar(0.5)
    slots = [t, r]
    assert E._slot_of(slots, t) == 0 and E._slot_of(slots, r) == 1
    for other in (torch.zeros(4), torch.zeros(4, dtype=torch.uint8), E.Scalar(0.5), 0.5, 3, None, "x"):
        with pytest.raises(ValueError):
            E._slot_of(slots, other)


@pytest.mark.gpu
def test_gradient_of_a_plain_number_is_zero(lib, dev):
    t = torch.ones(9, device=dev)
    g, z = E.vjp([torch.empty_like(t)], [E.Table(t) * E.Table(t)], [t], [t, 0.25])
    assert (g == 2.0).all() and z.item() == 0.0 and z.dtype == torch.float64
