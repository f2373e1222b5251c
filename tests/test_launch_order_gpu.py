"""Kernels that may be launched before the stream's previous kernel has ended see
all that it wrote, and write nothing it still reads: chains of calls that feed one
another, at sizes of a part of a wave of blocks and of several, on the default
and on another stream, with torch's own kernels between, and from a captured
graph of two streams.  Equal to the same calls with a synchronisation after each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(lib, step, n, dev, prec, table):
    g = torch.Generator(device=dev)
    g.manual_seed(n)

    def u(a, b):
        return torch.rand(n, device=dev, generator=g) * (b - a) + a

    S, K, T, V = u(5, 30), u(5, 30), u(0.25, 10), u(0.1, 0.6)
    a, b, c, d = (torch.zeros(n, device=dev) for _ in range(4))
    kw = dict(precision=prec)

    def price(s, k, o, p):
        if table:
            lib.blackscholes(s, k, T, o, p, 0.02, sigma=V, **kw)
        else:
            lib.blackscholes(s, k, T, o, p, 0.02, sigma_s=0.3, **kw)
        step()

    for _ in range(6):
        price(S, K, a, b)          # a, b from S, K
        price(a, b, c, d)          # c, d from what was just written
        price(c, K, a, b)          # over what the last call read
        S.add_(a, alpha=0.125)     # a torch kernel between
        step()
        price(S, S, S, d)          # in place
        S.add_(5.0)
        step()
    return [t.clone() for t in (S, a, b, c, d)]


@pytest.mark.parametrize("table", [False, True], ids=["one_volatility", "volatility_table"])
@pytest.mark.parametrize("prec", ["fast", "nt2"])
@pytest.mark.parametrize("n", [3, 4096, 300_001, 1 << 20, 3_000_001])
def test_chained_calls(lib, dev, n, prec, table):
    p = lib.PREC_NT2 if prec == "nt2" else lib.PREC_FAST
    want = _chain(lib, torch.cuda.synchronize, n, dev, p, table)
    got = _chain(lib, lambda: None, n, dev, p, table)
    with torch.cuda.stream(torch.cuda.Stream()):
        other = _chain(lib, lambda: None, n, dev, p, table)
    torch.cuda.synchronize()
    for w, x, y in zip(want, got, other):
        assert torch.equal(w.view(torch.int32), x.view(torch.int32))
        assert torch.equal(w.view(torch.int32), y.view(torch.int32))


def test_chained_calls_in_a_graph_of_two_streams(lib, dev):
    n = 1 << 20
    S, K, T = (torch.rand(n, device=dev) * 20 + 5 for _ in range(3))
    bufs = [torch.zeros(n, device=dev) for _ in range(8)]

    def calls(side):
        main = torch.cuda.current_stream()
        lib.blackscholes(S, K, T, bufs[0], bufs[1], 0.02, sigma_s=0.3)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            lib.blackscholes(bufs[0], K, T, bufs[2], bufs[3], 0.02, sigma_s=0.3)
        lib.blackscholes(bufs[1], K, T, bufs[4], bufs[5], 0.02, sigma_s=0.3)
        main.wait_stream(side)
        lib.blackscholes(bufs[2], bufs[4], T, bufs[6], bufs[7], 0.02, sigma_s=0.3)

    side = torch.cuda.Stream()
    calls(side)
    torch.cuda.synchronize()
    want = [b.clone() for b in bufs]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls(side)
    for _ in range(5):
        for b in bufs:
            b.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for b, w in zip(bufs, want):
            assert torch.equal(b.view(torch.int32), w.view(torch.int32))


def _folds_chain(lib, step, rows, cols, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(rows)
    t = torch.rand(rows * cols, device=dev, generator=g) * 4 + 1
    seen = []
    for k in range(3):
        for op in ("mean", "stdev", "max"):
            down = lib.fold(t, 1, rows, cols, op)        # along columns
            step()
            across = lib.fold(t, rows, cols, 1, op)      # along rows
            step()
            both = lib.fold(down, 1, cols, 1, op)        # of what was just written
            step()
            t[:cols] = down                              # feed the next calls
            t[-rows:] = across
            t[0] += both[0]
            step()
            seen += [down, across, both]
        for shape in ((1, rows, cols), (rows, cols, 1), (1, rows * cols, 1)):
            m = lib.median(t, *shape)
            step()
            t[k:k + m.numel()] += m * 0.25
            step()
            seen.append(m)
    return [s.clone() for s in seen + [t]]


@pytest.mark.parametrize("rows,cols", [(40, 60), (3000, 17), (1500, 1100), (300, 3001), (50000, 4)])
def test_chained_folds_and_medians(lib, dev, rows, cols):
    want = _folds_chain(lib, torch.cuda.synchronize, rows, cols, dev)
    got = _folds_chain(lib, lambda: None, rows, cols, dev)
    torch.cuda.synchronize()
    for w, x in zip(want, got):
        assert torch.equal(w.view(torch.int32), x.view(torch.int32))
