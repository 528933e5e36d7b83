"""The two evaluation kernels against each other and the FP64 oracle: sums of one
warp (as many points as fill the GPU's warps once) and sums shared among warps
(few points).  The launches say which ran: a shared sum is added up by a second
kernel.  Both give the same bits, at every dimension where the kernels' forms
change (unrolled subtrees, loops) and with limits that cut rows and walks."""
import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs
from conftest import check_eval
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _evaluate(g, X, out, m):
    before = _lib.kernel_launches()
    g.evaluate_device(X, out, m)
    g.sync()
    return _lib.kernel_launches() - before


# segments: 16, 16, 32 in 2 parts, 48 in 3, 80 in 5, 16 .. 80 above 12 dims
@pytest.mark.parametrize("d,n,lim", [
    (4, 14, None), (6, 9, [8, 2, 5, 8, 8, 3]), (5, 12, None), (10, 7, None), (9, 8, None), (12, 6, None),
    (13, 4, None), (13, 6, None), (13, 7, [6, 1, 3, 6, 2, 6, 1, 4, 6, 6, 3, 6, 6]), (14, 6, None), (15, 5, None),
    (16, 5, None), (16, 6, [5, 5, 1, 5, 0, 5, 5, 2, 5, 5, 5, 5, 4, 1, 5, 2]), (17, 5, None), (20, 5, None)])
def test_shared_sums_equal_whole_sums(cuda, d, n, lim):
    import torch
    g = sg.Grid(d, n, lim)
    g.set_values(inputs.uniform01(d + n, g.num_points) * 2 - 1)
    g.hierarchize()
    g.set_option(sg.SG_OPT_EVAL_SORT, 0)
    m = torch.cuda.get_device_properties(cuda).multi_processor_count * 16 * 64
    X = inputs.uniform_points(3 * d + n, m, d)
    X[5], X[70] = 1.5, np.nan
    X[7] = 2.0 ** -20
    Xd = torch.from_numpy(X).to(cuda)
    whole = torch.empty(m, device=cuda)
    _evaluate(g, Xd, whole, 1)  # the block layout
    assert _evaluate(g, Xd, whole, m) == 1
    for k in (1, 63, 64, 65, 1000):
        out = torch.full((k,), 7.0, device=cuda)
        assert _evaluate(g, Xd, out, k) == 2
        assert torch.equal(out.view(torch.int32), whole[:k].view(torch.int32)), k
    w = whole.cpu().numpy()
    assert w[5] == 0.0 and np.isnan(w[70])
    idx = np.concatenate([[0, 7], np.arange(100, 140)])
    check_eval(w[idx], Oracle(d, n, lim).evaluate_f64(g.get_values().astype(np.float64), X[idx]), f"d={d} n={n}",
               per_point=False)


@pytest.mark.parametrize("d,n,level,value", [(2, 7, (2, 3), np.inf), (3, 6, (1, 0, 4), -np.inf), (4, 6, (2, 1, 0, 2), np.inf),
                                             (13, 3, (0,) * 12 + (2,), np.inf), (6, 7, (0, 1, 0, 2, 0, 3), np.nan)])
def test_a_non_finite_surplus_stays_in_its_cell(cuda, d, n, level, value):
    """Inside its basis function's support the sum is not finite, every other
    point is as without it."""
    g = sg.Grid(d, n)
    index = [(1 << l) // 2 for l in level]
    at = g.gp2idx(level, index)
    s = (inputs.uniform01(d, g.num_points) * 2 - 1).astype(np.float32)
    X = inputs.uniform_points(7, 4000, d)
    lo = np.array(index) / 2.0 ** np.array(level)
    width = 1.0 / 2.0 ** np.array(level)
    X[:500] = (lo + width * (0.05 + 0.9 * inputs.uniform_points(8, 500, d))).astype(np.float32)
    inside = ((X > lo) & (X < lo + width)).all(axis=1)
    away = ((X < lo) | (X > lo + width)).any(axis=1)
    s[at] = 0.0
    g.set_values(s)
    clean = g.evaluate(X)
    s[at] = value
    g.set_values(s)
    out = g.evaluate(X)
    assert inside.sum() >= 500 and away.sum() > 100
    assert not np.any(np.isfinite(out[inside]))
    assert np.array_equal(out[away].view(np.uint32), clean[away].view(np.uint32))


def test_segments_keep_their_compensation(cuda):
    """2^24 + 1 inside one segment and -2^24 in another: the 1, which no float
    beside 2^24 holds, survives the segment's end, in whole and in shared sums."""
    import torch
    d, n = 10, 7
    g = sg.Grid(d, n)
    s = np.zeros(g.num_points, np.float32)
    # at x = 1/4 the hats are 1/2 at level 0, 1 at level 1 and 0 above; the first
    # two are neighbours in the walk, in a subtree that no segment divides
    for levels, value in (((1, 1, 1, 0, 0, 0, 0, 0, 0, 0), 2.0 ** 24), ((1, 1, 1, 0, 0, 1, 0, 0, 0, 0), 1.0),
                          ((0,) * 10, -2.0 ** 24)):
        s[g.gp2idx(levels, (0,) * d)] = value * 2.0 ** (d - sum(levels))
    g.set_values(s)
    m = torch.cuda.get_device_properties(cuda).multi_processor_count * 16 * 64
    X = torch.full((m, d), 0.25, device=cuda)
    for k in (1, 1000, m):
        out = torch.empty(k, device=cuda)
        g.evaluate_device(X, out, k)
        g.sync()
        assert bool((out == 1.0).all()), (k, float(out[0]))
