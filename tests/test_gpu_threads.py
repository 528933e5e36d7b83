"""Host threads with a handle each: grids and batches of very different size,
whose launches ask for very different amounts of shared memory, hierarchized at
the same time give the bits that they give alone."""
import threading

import numpy as np
import pytest

import adaptive_sparse_grid_bench_b200 as sg
from adaptive_sparse_grid_bench_b200 import _lib, inputs

pytestmark = pytest.mark.gpu


def _run_all(workers):
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in workers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


# passes of 2 and 3 dims in units of 2 to 100 KB; single-dim sweeps (n = 12)
@pytest.mark.parametrize("shapes,precision", [
    ([(6, 7), (10, 9), (8, 8), (7, 10)], "fp32"), ([(6, 7), (9, 8), (8, 8), (7, 9)], "fp64"),
    ([(5, 4), (8, 6), (20, 4), (12, 5)], "fp32"), ([(3, 12), (2, 7), (4, 11), (3, 5)], "fp32")])
def test_threads_hierarchize_their_own_grids(cuda, shapes, precision):
    def worker(d, n):
        def run():
            g = sg.Grid(d, n)
            g.precision = precision
            v = inputs.uniform01(d + n, g.num_points) * 2 - 1
            g.set_values(v)
            g.hierarchize()
            want = g.get_values().view(np.uint32)
            for _ in range(40):
                g.set_values(v)
                g.hierarchize()
                assert np.array_equal(g.get_values().view(np.uint32), want)
            g.close()
        return run
    _run_all([worker(d, n) for d, n in shapes for _ in range(2)])


def test_threads_hierarchize_their_own_batches(cuda):
    def worker(shapes):
        def run():
            b = sg.Batch([s[0] for s in shapes], [s[1] for s in shapes])
            b.set_option(_lib.SG_OPT_USE_GRAPH, 0)
            v = inputs.uniform01(len(shapes), b.num_values) * 2 - 1
            b.set_values(v)
            b.hierarchize()
            want = b.get_values().view(np.uint32)
            for _ in range(60):
                b.set_values(v)
                b.hierarchize()
                assert np.array_equal(b.get_values().view(np.uint32), want)
            b.close()
        return run
    # grids of 1,023 points and below, and of 4,097 to 25,000
    _run_all([worker(w) for w in ([(2, 5), (3, 4)], [(4, 6), (2, 9)], [(5, 6), (6, 5)], [(3, 3)] * 3) for _ in range(2)])
