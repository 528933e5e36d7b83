"""Evaluations of one grid that overlap on several streams, and evaluations
recorded into CUDA graphs: whichever way a point's sum is added up, each call
gives the bits that it gives alone."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs

pytestmark = pytest.mark.gpu


def _grid(d, n):
    g = sg.Grid(d, n)
    g.set_values(inputs.uniform01(d * n, g.num_points) * 2 - 1)
    g.hierarchize()
    return g


def _points(cuda, seed, m, d):
    import torch
    return torch.from_numpy(inputs.uniform_points(seed, m, d)).to(cuda)


def _bits(t):
    import torch
    return t.view(torch.int32)


# shared by segments and by parts; one point (never ordered) at the default options
@pytest.mark.parametrize("d,n,m,sort", [(10, 8, 1000, 0), (10, 8, 60_000, 0), (6, 12, 700, 0), (10, 8, 1, 1)])
def test_two_streams_on_one_grid(cuda, d, n, m, sort):
    import torch
    g = _grid(d, n)
    g.set_option(sg.SG_OPT_EVAL_SORT, sort)
    streams = [torch.cuda.Stream() for _ in range(3)]
    X = [_points(cuda, 10 + i, m, d) for i in range(len(streams))]
    alone = [torch.empty(m, device=cuda) for _ in streams]
    for x, o in zip(X, alone):
        g.evaluate_device(x, o)
    g.sync()
    torch.cuda.synchronize()
    outs = [[torch.full((m,), np.nan, device=cuda) for _ in streams] for _ in range(8)]
    torch.cuda.synchronize()
    for row in outs:
        for x, o, st in zip(X, row, streams):
            g.evaluate_device(x, o, stream=st)
    torch.cuda.synchronize()
    for row in outs:
        for o, a in zip(row, alone):
            assert torch.equal(_bits(o), _bits(a))


def test_smaller_call_after_a_larger_one_under_capture(cuda):
    """What a call needs never grows as its points get fewer: after a call with
    many points, one with fewer records into a graph, and the graph gives the
    same bits after further calls of other sizes."""
    import torch
    d, n = 10, 8
    g = _grid(d, n)
    X = _points(cuda, 3, 100_000, d)
    want = torch.empty(100_000, device=cuda)
    g.evaluate_device(X, want)
    g.sync()
    out = torch.empty(50_000, device=cuda)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.evaluate_device(X, out, 50_000, torch.cuda.current_stream())
    other = torch.empty(100_000, device=cuda)
    for m in (1000, 20_000, 70_000):
        g.evaluate_device(X, other, m)
    g.sync()
    for _ in range(2):
        out.fill_(np.nan)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(_bits(out), _bits(want[:50_000]))


def test_captured_evaluations_share_their_sums(cuda):
    """A captured call keeps its sums in memory of its own: two graphs of one grid
    and an eager call run side by side.  Where the handle has no more room for
    such memory the call takes whole sums: one launch less, the same bits."""
    import torch
    d, n, m = 10, 8, 60_000
    g = _grid(d, n)
    g.set_option(sg.SG_OPT_EVAL_SORT, 0)
    X = [_points(cuda, 20 + i, m, d) for i in range(3)]
    want = [torch.empty(m, device=cuda) for _ in X]
    for x, o in zip(X, want):
        g.evaluate_device(x, o)
    g.sync()
    got = [torch.empty(m, device=cuda) for _ in X]
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    for k, graph in enumerate(graphs):
        with torch.cuda.graph(graph):
            before = _lib.kernel_launches()
            g.evaluate_device(X[k], got[k], m, torch.cuda.current_stream())
            assert _lib.kernel_launches() - before == 2  # the sums, and adding them up
    streams = [torch.cuda.Stream() for _ in X]
    torch.cuda.synchronize()
    for _ in range(5):
        for k, st in enumerate(streams):
            with torch.cuda.stream(st):
                if k < len(graphs):
                    graphs[k].replay()
                else:
                    g.evaluate_device(X[k], got[k], m, st)
    torch.cuda.synchronize()
    for o, w in zip(got, want):
        assert torch.equal(_bits(o), _bits(w))
    # 128 segments x 10,000 points x 8 bytes: room for 12 more beside these two
    launches = []
    for _ in range(30):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            before = _lib.kernel_launches()
            g.evaluate_device(X[0], got[0], 10_000, torch.cuda.current_stream())
            launches.append(_lib.kernel_launches() - before)
        got[0].fill_(np.nan)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(_bits(got[0][:10_000]), _bits(want[0][:10_000]))
    assert launches[0] == 2 and launches[-1] == 1


def test_memory_of_shared_sums_is_given_back(cuda):
    import torch

    def cycle():
        g = _grid(10, 8)
        x, o = _points(cuda, 5, 50_000, 10), torch.empty(50_000, device=cuda)
        g.evaluate_device(x, o)
        g.sync()
        used = torch.cuda.mem_get_info()[0]
        g.close()
        torch.cuda.synchronize()
        return used, torch.cuda.mem_get_info()[0]

    cycle()  # the allocator's own caches
    first, second = cycle(), cycle()
    assert first[1] == second[1] and first[1] > first[0]
