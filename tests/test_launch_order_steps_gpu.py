"""A sigma-delta step whose frame is what the kernel just before wrote: labels of
another step (a fold, which lets the next kernel line up early, between them or
not), prices seen as bytes.  Equal to the same calls with a synchronisation after
each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(lib, step, n, dev, off):
    g = torch.Generator(device=dev)
    g.manual_seed(n)
    scene = torch.randint(0, 256, (n,), device=dev, generator=g, dtype=torch.uint8)
    room = [torch.zeros(n + 16, dtype=torch.uint8, device=dev)[off:off + n] for _ in range(8)]
    b1, v1, l1, b2, v2, l2, b3, l3 = room
    table = torch.rand(1 << 20, device=dev, generator=g)
    small = torch.rand(4096, device=dev, generator=g)
    m = (n + 3) // 4
    S, K, T = (torch.rand(m, device=dev, generator=g) * 20 + 5 for _ in range(3))
    call, put = torch.zeros(m, device=dev), torch.zeros(m, device=dev)
    seen = []
    for k in range(6):
        lib.sigmadelta(scene, b1, v1, l1)
        step()
        if k % 3:  # one kernel, or a fold and the one that combines it
            lib.fold(small if k % 3 == 1 else table, 1, 4096 if k % 3 == 1 else 1 << 20, 1, "sum")
            step()
        lib.sigmadelta(l1, b2, v2, l2)
        step()
        lib.blackscholes(S, K, T, call, put, 0.02, sigma_s=0.2 + 0.1 * k)
        step()
        lib.sigmadelta(call.view(torch.uint8)[:n], b3, v2, l3)
        step()
        scene = scene + l2 // 2 + 3
        S += 0.5
        step()
        seen += [t.clone() for t in (l1, l2, l3, b2, b3, v2)]
    return seen


@pytest.mark.parametrize("n,off", [(1920 * 1080, 0), (640 * 360, 0), (100, 0), (1921 * 541, 0), (1920 * 1080, 3)])
def test_steps_on_what_was_just_written(lib, dev, n, off):
    want = _chain(lib, torch.cuda.synchronize, n, dev, off)
    got = _chain(lib, lambda: None, n, dev, off)
    torch.cuda.synchronize()
    for w, x in zip(want, got):
        assert torch.equal(w, x)
