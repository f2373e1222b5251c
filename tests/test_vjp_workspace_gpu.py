"""A scalar's gradient with the workspace asked for, and with one for half of the
blocks (a partial sum for every 1024 elements); less is refused."""
import ctypes

import pytest
import torch

from nt2_gb300 import expr as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 513, 1025, 100003, 700001, 2000003])
def test_half_the_workspace(lib, dev, n):
    x = torch.rand(n, device=dev) + 0.5
    out, ct, r = torch.empty_like(x), torch.ones_like(x), E.Scalar(0.25)
    prog, slots = E.compile_program([out], [E.exp(E.Table(x) * r)])
    args, _ = E._args_of(slots)
    ns, L = len(slots), lib.load()
    cts, grads = (ctypes.c_void_p * ns)(), (ctypes.c_void_p * ns)()
    cts[E._slot_of(slots, out)] = ct.data_ptr()
    asked = ctypes.c_size_t()
    lib.check(L.nt2g_program_vjp_workspace_size(prog.handle, n, ctypes.byref(asked)))
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    half = 8 * min((n + 1023) // 1024, 8 * sms)
    assert half <= asked.value <= 2 * half
    ws = torch.empty(asked.value + 16, dtype=torch.uint8, device=dev)
    res = []
    for size in (asked.value, half):
        sums = torch.zeros(ns, dtype=torch.float64, device=dev)
        lib.check(L.nt2g_program_vjp(prog.handle, args, ns, n, cts, grads, lib._ptr(sums), lib.PREC_FAST, lib._ptr(ws), size,
                                     lib._stream()))
        res.append(sums[E._slot_of(slots, r)].item())
    exact = (x.double() * torch.exp(x.double() * 0.25)).sum().item()
    # each adjoint rounds a few times in float; the sums agree to FP64's rounding of n addends
    assert abs(res[0] - res[1]) <= 2.0 ** -50 * n ** 0.5 * abs(exact) and abs(res[0] - exact) <= 1e-6 * exact
    assert L.nt2g_program_vjp(prog.handle, args, ns, n, cts, grads, lib._ptr(ws), lib.PREC_FAST, lib._ptr(ws), 0,
                              lib._stream()) == lib.ERR_INVALID
