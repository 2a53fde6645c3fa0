"""The cache of nebo_heat_run's graphs: runs whose arguments keep changing hold a bounded number of
graphs and at most 128 MiB of scratch, and give the bits of the same run without a graph, for a new
graph, a repeated one, one that was dropped and is made again, and one that found no room; graphs of
several threads, and one graph from several threads, too."""
import threading

import pytest
import torch

import spatialops_gb300 as N

pytestmark = pytest.mark.gpu


class Case:
    def __init__(self, n, seed=0):
        self.T, self.tmp, self.lam = (N.Field("SVol", n, 1) for _ in range(3))
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.T0 = torch.randn(self.T.tensor.shape, generator=g, device="cuda", dtype=torch.float64)
        self.lam.tensor.uniform_(0.5, 1.0, generator=g)

    def run(self, steps, dt, graph, stream=None):
        self.T.tensor.copy_(self.T0)
        N.heat_run(self.T, self.tmp, self.lam, steps, dt, use_graph=graph, stream=stream)
        return self.T.tensor.clone()


def test_many_time_steps():
    c = Case((24, 20, 16))
    dts = [0.05 * (1 + 1e-6 * k) for k in range(1700)]
    for k, dt in enumerate(dts):
        got = c.run(3 + k % 2, dt, True)
        if k % 100 == 0:
            assert torch.equal(got, c.run(3 + k % 2, dt, False))
            assert torch.equal(got, c.run(3 + k % 2, dt, True))
    assert torch.equal(c.run(3, dts[0], True), c.run(3, dts[0], False))


def test_scratch_is_bounded():
    c = Case((64, 60, 56))  # 5.7 MB of scratch a graph
    want = [c.run(4, 0.05 * (1 + 1e-6 * k), False) for k in (0, 30)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    got = []
    for k in range(31):
        r = c.run(4, 0.05 * (1 + 1e-6 * k), True)
        if k in (0, 30):
            got.append(r)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= (128 << 20) + (64 << 20)
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_field_without_room():
    c = Case((120, 118, 116))
    assert torch.equal(c.run(5, 0.05, True), c.run(5, 0.05, False))


def test_threads():
    own = [Case((40 + i, 33, 30), i) for i in range(4)]
    want = [c.run(8, 0.05, False) for c in own]
    shared = Case((64, 48, 40), 9)
    shared_want = shared.run(8, 0.05, False)
    torch.cuda.synchronize()
    bad, turn = [], threading.Lock()

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for k in range(60):
                if not torch.equal(own[i].run(8, 0.05, True, s), want[i]):
                    bad.append(i)
                own[i].run(8, 0.05 * (1 + 1e-6 * (k % 7)), True, s)
                with turn:  # one run of the shared fields at a time, from every thread and stream
                    if not torch.equal(shared.run(8, 0.05, True, s), shared_want):
                        bad.append("shared")
                    s.synchronize()

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
