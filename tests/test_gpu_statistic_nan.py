"""NaN in the refinement statistic: a run of 32 NaN, or a whole smaller
subspace of them, makes the subspace's maximum NaN at every level sum (a value
that diverged is not reported as converged); single NaN values are passed over."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import inputs

pytestmark = pytest.mark.gpu


def _subspace_sums(g):
    dp, _ = g.tables()
    return np.repeat(np.arange(g.n), dp[g.d - 1].astype(np.int64))


def _expected(v, sums):
    out, at = [], 0
    for s in sums:
        a = np.abs(v[at:at + (1 << s)])
        at += 1 << s
        runs = a.reshape(-1, min(32, a.size))
        # fmax passes NaN over: the maximum of a run is NaN only if all of it is
        m = np.fmax.reduce(runs, axis=1)
        out.append(np.nan if np.isnan(m).any() else m.max())
    return np.array(out, np.float32)


# level sums 0..12 (one atomic from 11 on); one to many subspaces per 1024 values
@pytest.mark.parametrize("d,n", [(1, 13), (2, 12), (4, 9)])
def test_nan_in_the_statistic(cuda, d, n):
    g = sg.Grid(d, n)
    sums = _subspace_sums(g)
    start = np.concatenate([[0], np.cumsum(1 << sums)])
    base = inputs.uniform01(d + n, g.num_points) * 2 - 1
    for fill in ("all", "one run", "crooked run", "last value", "all but one"):
        v = base.copy()
        for q in range(0, len(sums), 3):  # every third subspace
            a = v[start[q]:start[q + 1]]
            if fill == "all":
                a[:] = np.nan
            elif fill == "one run":
                a[-32:] = np.nan
            elif fill == "crooked run" and a.size > 32:
                a[16:48] = np.nan
            elif fill == "last value":
                a[-1] = np.nan
            elif fill == "all but one":
                a[1:] = np.nan
        g.set_values(v)
        got, want = g.subspace_maxabs(), _expected(v, sums)
        assert np.array_equal(np.isnan(got), np.isnan(want)), fill
        ok = ~np.isnan(want)
        assert np.array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32)), fill
