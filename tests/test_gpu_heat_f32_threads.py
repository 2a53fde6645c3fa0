"""FP32 heat steps from two host threads at once, one on wide rows and one on narrow ones: the kernel's
shared-memory limit is the same for both, so no launch is refused, and each ends with the bits of the
same steps alone."""
import threading

import pytest
import torch

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


def _fields(nx):
    n = (nx, 12, 6)
    T, tmp, lam = (N.Field("SVol", n, 1, dtype="f32") for _ in range(3))
    T.tensor.normal_(generator=torch.Generator(device="cuda").manual_seed(nx))
    lam.tensor.fill_(1.0)
    return T, tmp, lam


def _run(nx, count, s):
    T, tmp, lam = _fields(nx)
    s.wait_stream(torch.cuda.current_stream())
    for _ in range(count):
        N.heat_run(T, tmp, lam, 100, 0.1, use_graph=False, stream=s)
    s.synchronize()
    return T.tensor.cpu()


def test_two_threads_of_different_widths():
    widths = (1000, 64)
    alone = [_run(nx, 40, torch.cuda.Stream()) for nx in widths]
    got, failed = [None, None], []

    def work(i):
        try:
            got[i] = _run(widths[i], 40, torch.cuda.Stream())
        except Exception as e:  # a refused launch
            failed.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not failed
    assert all(torch.equal(a, b) for a, b in zip(alone, got))
