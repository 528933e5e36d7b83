"""The caller's buffers of sg_set_values_device and sg_get_values_device: the
kernel moves between this GPU's float-aligned buffers only; every other buffer
that a copy can reach is copied, with the same values."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs

pytestmark = pytest.mark.gpu


def _round_trip(g, src, dst):
    """Launches of the library's own kernels while values move in and out."""
    before = _lib.kernel_launches()
    g.set_values_device(src)
    g.get_values_device(dst)
    g.sync()
    return _lib.kernel_launches() - before


@pytest.mark.parametrize("d,n", [(1, 1), (4, 8), (10, 6)])
def test_buffers_off_the_float_grid_are_copied(cuda, d, n):
    import torch
    g = sg.Grid(d, n)
    v = inputs.uniform01(d + n, g.num_points) * 2 - 1
    raw = torch.from_numpy(v.view(np.uint8).copy()).to(cuda)
    for shift in (0, 1, 2, 6):
        src = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device=cuda)
        dst = torch.full_like(src, 7)
        src[shift:shift + raw.numel()] = raw
        launches = _round_trip(g, src[shift:], dst[shift:])
        assert launches == (2 if shift % 4 == 0 else 0), shift
        assert torch.equal(dst[shift:shift + raw.numel()], raw)
        assert bool((dst[:shift] == 7).all()) and bool((dst[shift + raw.numel():] == 7).all())
        assert np.array_equal(g.get_values(), v)


def test_pinned_host_buffers_are_copied(cuda):
    import torch
    g = sg.Grid(5, 7)
    v = inputs.uniform01(5, g.num_points) * 2 - 1
    src = torch.from_numpy(v.copy()).pin_memory()
    dst = torch.empty(g.num_points).pin_memory()
    assert _round_trip(g, src, dst) == 0
    assert np.array_equal(dst.numpy(), v) and np.array_equal(g.get_values(), v)
