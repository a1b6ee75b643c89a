"""Calls of odd sizes on one plan from several streams and host threads: the padded copies
they are staged through are ordered, so results are those of calls one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(gtb, subsets):
    L = gtb._lib
    n, W, H, P = (75, 70, 61), 131, 93, 24
    g = L.CbctGeometry(1000.0, 1500.0, W * 1.1, H * 1.1, W, H, n[0], n[1], n[2], float(n[0]), float(n[1]), float(n[2]), 1.5)
    return gtb.Plan(g, (3.0 + np.arange(P) * 15.0).astype(np.float32), np.zeros((P, 2), np.float32), subsets)


def _inputs(cuda, plan, k):
    import torch
    gen = torch.Generator(device=cuda)
    gen.manual_seed(k)
    return torch.rand(plan.proj_shape(k % 2), generator=gen, device=cuda), torch.rand(plan.vol_shape, generator=gen, device=cuda)


@pytest.mark.parametrize("threads", [False, True])
def test_two_streams(gtb, cuda, threads):
    import torch
    plan = _plan(gtb, np.array([12, 12], np.int32))
    data = [_inputs(cuda, plan, k) for k in range(8)]
    want = []
    for k, (proj, vol) in enumerate(data):
        want.append((plan.backproject(proj, torch.empty_like(vol), k % 2), plan.forward(vol, torch.empty_like(proj), k % 2)))
    torch.cuda.synchronize()
    got = [(torch.empty_like(v), torch.empty_like(p)) for p, v in data]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()

    def work(t):
        for _ in range(5):
            for k in range(t, 8, 4):
                plan.backproject(data[k][0], got[k][0], k % 2, stream=streams[t].cuda_stream)
                plan.forward(data[k][1], got[k][1], k % 2, stream=streams[t].cuda_stream)

    if threads:
        ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for t in range(4):
            work(t)
    torch.cuda.synchronize()
    assert plan.read_flags() == (0, 0)
    for a, b in zip(got, want):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_streams_of_one_capture(gtb, cuda):
    """Two branches of one captured graph, and eager calls before and after."""
    import torch
    plan = _plan(gtb, np.array([12, 12], np.int32))
    data = [_inputs(cuda, plan, k) for k in range(2)]
    want = [plan.backproject(p, torch.empty_like(v), k) for k, (p, v) in enumerate(data)]
    got = [torch.empty_like(v) for _, v in data]
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        plan.backproject(data[0][0], got[0], 0, stream=main.cuda_stream)
        with torch.cuda.stream(side):
            plan.backproject(data[1][0], got[1], 1, stream=side.cuda_stream)
        main.wait_stream(side)
    for _ in range(3):
        for v in got:
            v.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    again = plan.backproject(data[0][0], torch.empty_like(got[0]), 0, stream=side.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(again, want[0])
