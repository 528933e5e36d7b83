"""Hierarchization passes of one, two and three dims (and the single-dim sweeps
around them): surpluses bit-identical to hierarchize0 (c:557-571) in FP32 and
to the FP64 oracle rounded once, on shapes whose units have 1, 2, 4 and many
cells, cells contiguous or not, and limits that cut the units short."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,lim", [
    (4, 6, None), (5, 6, None), (7, 6, None), (20, 4, None),                       # three dims per pass, rests of 1 and 2
    (5, 2, None), (9, 3, [0, 2, 0, 1, 2, 0, 2, 2, 1]), (7, 6, [5, 5, 0, 5, 5, 0, 5]),  # budget 1; dims without levels
    (5, 8, None), (6, 7, [6, 2, 5, 6, 6, 1]), (8, 8, None), (6, 10, None), (7, 9, [8, 1, 8, 8, 3, 8, 8]),  # two dims
    (5, 11, None), (4, 12, [11, 9, 11, 10])])                                        # single-dim sweeps and passes mixed
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_passes_bit_exact(cuda, d, n, lim, precision):
    o = Oracle(d, n, lim)
    g = sg.Grid(d, n, lim)
    g.precision = precision
    v = inputs.uniform01(13 * d + n, g.num_points) * 2 - 1
    g.set_values(v)
    g.hierarchize()
    want = (o.hierarchize_f32(v) if precision == "fp32"
            else o.hierarchize_f64(v.astype(np.float64)).astype(np.float32))
    assert np.array_equal(g.get_values().view(np.uint32), want.view(np.uint32))


def test_options_changed_on_a_live_grid(cuda):
    """The tables of another precision or sweep kernel are built when the option
    is set, and every setting gives the same FP32 bits."""
    d, n = 6, 8
    o = Oracle(d, n)
    g = sg.Grid(d, n)
    v = inputs.uniform01(3, g.num_points) * 2 - 1
    want = {"fp32": o.hierarchize_f32(v), "fp64": o.hierarchize_f64(v.astype(np.float64)).astype(np.float32)}
    for precision, kernel in (("fp32", 0), ("fp32", 2), ("fp64", 0), ("fp64", 2), ("fp32", 1), ("fp64", 1)):
        g.precision = precision
        g.set_option(sg.SG_OPT_HIER_KERNEL, kernel)
        g.set_values(v)
        g.hierarchize()
        assert np.array_equal(g.get_values().view(np.uint32), want[precision].view(np.uint32)), (precision, kernel)


def test_hierarchize_under_capture(cuda):
    """Nothing is allocated or copied by a hierarchization whose tables exist: it
    records into a CUDA graph, and the replay gives the same bits."""
    import torch
    g = sg.Grid(5, 8)
    v = torch.from_numpy(inputs.uniform01(4, g.num_points) * 2 - 1).to(cuda)
    out = torch.empty_like(v)
    g.set_values_device(v)
    g.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st = torch.cuda.current_stream()
        g.set_values_device(v, st)
        g.hierarchize_async(st)
        g.get_values_device(out, st)
    graph.replay()
    torch.cuda.synchronize()
    want = Oracle(5, 8).hierarchize_f32(v.cpu().numpy())
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
