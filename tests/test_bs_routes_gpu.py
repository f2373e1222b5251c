"""Black-Scholes from 2^22 options on: one float4 a thread for a single
volatility and for the NT2 policy, pipelined tiles of 1024 options for the fast
policy with a volatility table.  Sizes around the threshold, whole tiles and a
wave of blocks; the same bits as the same tables one element off a 16-byte
boundary, which go one option at a time, and no bounded wait gave up."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [False, True], ids=["one_volatility", "volatility_table"])
@pytest.mark.parametrize("prec", ["fast", "nt2"])
@pytest.mark.parametrize("n", [(1 << 22) - 1, 1 << 22, (1 << 22) + 1021, (1 << 22) + 1024 * 777 + 3, 9_000_002])
def test_large_batches_match_option_by_option(lib, dev, n, prec, table):
    p = lib.PREC_NT2 if prec == "nt2" else lib.PREC_FAST
    g = torch.Generator(device=dev)
    g.manual_seed(n)

    def u(a, b):
        return torch.rand(n, device=dev, generator=g) * (b - a) + a

    ins = [u(5, 30), u(1, 100), u(0.25, 10), u(0.1, 0.6)]
    off = [torch.empty(n + 1, device=dev)[1:].copy_(t) for t in ins]
    outs = []
    for t in (ins, off):
        c, q = torch.full_like(t[0], 7.0), torch.full_like(t[0], 7.0)
        lib.blackscholes(t[0], t[1], t[2], c, q, 0.02, precision=p, **(dict(sigma=t[3]) if table else dict(sigma_s=0.3)))
        outs.append((c, q))
    torch.cuda.synchronize()
    for a, b in zip(*outs):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    count = ctypes.c_uint64()
    lib.check(lib.load().nt2g_wait_timeouts(ctypes.byref(count)))
    assert count.value == 0
