"""Values to and from the device in the caller's compact order: every value lands
where it came from, whatever the sizes of the level groups and the alignment of
the caller's buffer (only float alignment is asked for)."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,lim", [(1, 1, None), (1, 4, None), (1, 16, None), (3, 7, [6, 2, 4]), (2, 5, [0, 0]),
                                     (5, 9, None), (20, 4, None), (10, 8, None)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_device_round_trip(cuda, d, n, lim, shift):
    import torch
    g = sg.Grid(d, n, lim)
    v = inputs.uniform01(d + n, g.num_points) * 2 - 1
    src = torch.zeros(g.num_points + shift, device=cuda)
    src[shift:] = torch.from_numpy(v).to(cuda)
    back = torch.full((g.num_points + shift + 1,), np.nan, device=cuda)
    g.set_values_device(src[shift:])
    g.get_values_device(back[shift:])
    g.sync()
    assert torch.equal(back[shift:shift + g.num_points], src[shift:])
    assert bool(torch.isnan(back[:shift]).all()) and bool(torch.isnan(back[-1]))
    assert np.array_equal(g.get_values(), v)  # the host copy, group by group, agrees
