"""Evaluation at the edges of its forms: rows of every length in the innermost
dim (one surplus, a pair, a linear piece per half cell), sums of one segment,
several, and several parts, added by one warp or shared among many, points
ordered or not.  Every way of adding a sum gives the same bits; values are
within the parity bound of the FP64 oracle: |u - u64| <= 1e-5 max|u64| + 2e-7
(c:1237-1274)."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs
from conftest import check_eval
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _grid(d, n, lim, seed):
    g = sg.Grid(d, n, lim)
    g.set_values(inputs.uniform01(seed, g.num_points) * 2 - 1)
    g.hierarchize()
    return g


# last dim with 1, 2, 3 and 16 levels; limits that cut the rows short
@pytest.mark.parametrize("d,n,lim", [(1, 1, None), (1, 2, None), (1, 3, None), (1, 16, None), (2, 12, None),
                                     (2, 12, [11, 0]), (3, 11, [10, 10, 1]), (3, 12, [2, 11, 2]), (4, 5, [4, 0, 4, 1]),
                                     (13, 4, None)])
def test_row_forms_vs_fp64_oracle(cuda, d, n, lim):
    g = _grid(d, n, lim, 31 * d + n)
    X = inputs.uniform_points(d + n, 1500, d)
    X[:4] = [[0.0] * d, [0.5] * d, [np.nextafter(np.float32(1), np.float32(0))] * d, [2.0 ** -20] * d]
    ref = Oracle(d, n, lim).evaluate_f64(g.get_values().astype(np.float64), X)
    check_eval(g.evaluate(X), ref, f"d={d} n={n} lim={lim}", per_point=False)


# segments per sum: 2, 16, 16 with limits, 32 in 2 parts, 64 in 4, 128 in 8; d
# above 12 (no unrolled subtrees); points on both sides of a warp's 64
@pytest.mark.parametrize("d,n,lim", [(4, 8, None), (4, 14, None), (6, 9, [8, 2, 5, 8, 8, 1]), (5, 12, None),
                                     (10, 7, None), (9, 8, None), (6, 14, [9, 9, 9, 3, 9, 9]), (14, 6, None)])
def test_shared_and_whole_sums_same_bits(cuda, d, n, lim):
    import torch
    g = _grid(d, n, lim, d + n)
    m = 180_000  # enough points for whole sums
    X = inputs.uniform_points(3 * d + n, m, d)
    X[5], X[70] = 1.5, np.nan
    Xd = torch.from_numpy(X).to(cuda)
    whole = torch.empty(m, device=cuda)
    g.evaluate_device(Xd, whole)
    g.sync()
    for sort in (1, 0):
        g.set_option(sg.SG_OPT_EVAL_SORT, sort)
        for k in (1, 63, 65, 1000, 20_000):
            out = torch.empty(k, device=cuda)
            g.evaluate_device(Xd, out, k)
            g.sync()
            assert torch.equal(out.view(torch.int32), whole[:k].view(torch.int32)), (sort, k)
    w = whole.cpu().numpy()
    assert w[5] == 0.0 and np.isnan(w[70])
    idx = np.arange(100, 160)
    check_eval(w[idx], Oracle(d, n, lim).evaluate_f64(g.get_values().astype(np.float64), X[idx]), "sample",
               per_point=False)


def test_fixed_scratch_limits(cuda):
    """The no-allocation call shares sums where its fixed array has room and
    falls back to whole sums where it has not, with the same bits."""
    import torch
    g = _grid(10, 8, None, 4)
    for m in (500, 40_000, _lib.SG_NOALLOC_MAX_POINTS):
        X = torch.from_numpy(inputs.uniform_points(m, m, 10)).to(cuda)
        a, b = torch.empty(m, device=cuda), torch.empty(m, device=cuda)
        g.evaluate_device(X, a)
        g.evaluate_device_noalloc(X, b)
        g.sync()
        assert torch.equal(a.view(torch.int32), b.view(torch.int32)), m


def test_batch_shares_like_single_grids(cuda):
    """A small batch shares the sums of its large grids, a large one does not:
    both give the single grids' bits."""
    import torch
    shapes = [(10, 7), (6, 9), (9, 7), (4, 6), (2, 9)]
    b = sg.Batch([s[0] for s in shapes], [s[1] for s in shapes])
    v = inputs.uniform01(8, b.num_values) * 2 - 1
    b.set_values(v)
    b.hierarchize()
    for counts in ([300, 700, 1, 0, 513], [300_000, 400_000, 300_000, 200_000, 100_000]):
        po = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        xs = [torch.from_numpy(inputs.uniform_points(50 + i, max(c, 1), d)[:c]).to(cuda)
              for i, (c, (d, _)) in enumerate(zip(counts, shapes))]
        out = torch.empty(int(po[-1]), device=cuda)
        b.evaluate_device(po, torch.cat([x.reshape(-1) for x in xs]), out)
        b.sync()
        for i, (d, n) in enumerate(shapes):
            if not counts[i]:
                continue
            one = sg.Grid(d, n)
            one.set_values(b.grid_values(v, i))
            one.hierarchize()
            want = torch.empty(counts[i], device=cuda)
            one.evaluate_device(xs[i], want)
            one.sync()
            assert torch.equal(out[po[i]:po[i + 1]].view(torch.int32), want.view(torch.int32)), (i, counts[i])


def test_infinite_surplus_stays_in_its_cell(cuda):
    """An infinite surplus spoils the sum inside its basis function's support
    (NaN: the compensated sum subtracts infinities) and leaves every other point
    alone, as adding level by level does."""
    n = 6
    g = sg.Grid(1, n)
    s = (inputs.uniform01(2, g.num_points) * 2 - 1).astype(np.float32)
    s[(1 << 3) - 1 + 2] = np.inf  # level 3, cell 2: support (0.25, 0.375)
    g.set_values(s)
    X = ((np.arange(4000, dtype=np.float64) + 0.5) / 4000).astype(np.float32).reshape(-1, 1)
    out = g.evaluate(X)
    inside = (X[:, 0] > 0.25) & (X[:, 0] < 0.375)
    assert not np.any(np.isfinite(out[inside]))
    f = s.astype(np.float64)
    f[(1 << 3) - 1 + 2] = 0.0
    check_eval(out[~inside], Oracle(1, n).evaluate_f64(f, X[~inside]), "outside", per_point=False)
