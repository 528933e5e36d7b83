"""What a small pool of grids holds: the cap is asked for no more than a grid's
values, its evaluation layout and its tables, plus 64 KB."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs

pytestmark = pytest.mark.gpu


# (d, n, cap): values and layout, 28 bytes and 12 per dim and subspace, 64 KB
@pytest.mark.parametrize("d,n,cap", [(20, 1, 65_936 + 304), (20, 2, 71_716 + 220), (10, 3, 77_528 + 40),
                                     (2, 5, 68_300 + 52), (4, 8, 370_552 + 136)])
def test_small_cap_takes_a_small_grid(cuda, d, n, cap):
    srv = sg.Server(cap, max_batch_points=1 << 12)
    gid = srv.add_grid(d, n, _lib.SG_FN_PROD4)
    x = inputs.uniform_points(d, 100, d)
    out, _ = srv.wait(srv.submit(gid, x))
    one = sg.Grid(d, n)
    one.sample_function(_lib.SG_FN_PROD4)
    one.hierarchize()
    assert np.array_equal(out.view(np.uint32), one.evaluate(x).view(np.uint32))
    st = srv.stats()
    assert st["resident_grids"] == 1 and st["evictions"] == 0 and 0 < st["bytes_in_use"] <= cap
    srv.close()
