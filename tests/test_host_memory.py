"""The library's host code over a CUDA runtime in host memory (fake_cuda.c): what
it allocates when an allocation fails, which streams its calls touch, and how
often it allocates.  No GPU."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

from adaptive_sparse_grid_bench_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "adaptive_sparse_grid_bench_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake")
    cc = ["gcc", "-O1", "-fPIC", "-std=gnu11", "-I", os.path.join(CUDA, "include"), "-I", CSRC]
    objs = []
    for src in [os.path.join(CSRC, f) for f in ("sgrid.c", "sgrid_batch.c", "sg_layout.c")] + [
            os.path.join(ROOT, "tests", "fake_cuda.c")]:
        objs.append(str(out / (os.path.basename(src)[:-2] + ".o")))
        subprocess.run(cc + ["-c", src, "-o", objs[-1]], check=True)
    names = subprocess.run(["nm"] + objs, check=True, capture_output=True, text=True).stdout
    wanted = set(re.findall(r" U (sgk_\w+)", names)) - set(re.findall(r" T (sgk_\w+)", names))
    empty = out / "empty.c"
    empty.write_text("".join(f"int {n}() {{ return 0; }}\n" for n in sorted(wanted)))
    lib = str(out / "libfake.so")
    # -Bsymbolic: its own CUDA runtime, whatever else the process has loaded
    subprocess.run(cc + ["-shared", "-Wl,-Bsymbolic", str(empty)] + objs + ["-o", lib, "-lpthread"], check=True)
    so = C.CDLL(lib)
    for name, (res, args) in _lib.SIGNATURES.items():
        if hasattr(so, name):
            getattr(so, name).restype, getattr(so, name).argtypes = res, args
    for name in ("live", "pool_live", "allocs", "frees", "legacy", "waits", "unsafe"):
        getattr(so, "fake_" + name).restype = C.c_long
    so.fake_fail.argtypes = [C.c_long]
    so.fake_capture.argtypes = [C.c_void_p]
    return so


class Grid:
    def __init__(self, so, d, n):
        self.so, self.h, self.d = so, C.c_void_p(), d
        assert so.sg_create(d, n, None, C.byref(self.h)) == _lib.SG_OK
        v = C.c_int64()
        so.sg_num_points(self.h, C.byref(v))
        self.values = np.zeros(v.value, np.float32)

    def set_values(self):
        return self.so.sg_set_values(self.h, self.values.ctypes.data)

    def hierarchize(self):
        return self.so.sg_hierarchize(self.h)

    def device_bytes(self):
        v = C.c_int64()
        self.so.sg_device_bytes(self.h, C.byref(v))
        return v.value

    def close(self):
        self.so.sg_destroy(self.h)


def _until_no_failure(fake, attempt):
    """Calls attempt() with its first, second, ... allocation failing until none
    does; yields after every failure."""
    k = 0
    while True:
        fake.fake_fail(k)
        r = attempt()
        fake.fake_fail(-1)
        if r == _lib.SG_OK:
            return
        assert r == _lib.SG_ERR_NOMEM, k
        k += 1
        yield k


SHAPES = [(6, 6), (3, 8), (5, 11)]  # passes of several dims; single-dim sweeps; both


@pytest.mark.parametrize("d,n", SHAPES)
def test_failed_set_up_leaves_nothing_allocated(fake, d, n):
    start = fake.fake_live()
    g = Grid(fake, d, n)
    fails = 0
    for fails in _until_no_failure(fake, g.set_values):
        assert fake.fake_live() == start and g.device_bytes() == 0
    assert fails > 5
    g.close()
    assert fake.fake_live() == start


@pytest.mark.parametrize("d,n", SHAPES)
@pytest.mark.parametrize("option,value", [(_lib.SG_OPT_HIER_PRECISION, _lib.SG_HIER_FP64),
                                          (_lib.SG_OPT_HIER_KERNEL, 2)])
def test_failed_tables_are_not_lost(fake, d, n, option, value):
    """Tables of another option, built on a live grid: an attempt that fails
    halfway and is made again leaves nothing behind that is not freed with the
    grid."""
    start, k = fake.fake_live(), 0
    while True:
        g = Grid(fake, d, n)
        assert g.set_values() == _lib.SG_OK
        fake.fake_fail(k)
        r = fake.sg_set_option(g.h, option, value)
        if r == _lib.SG_OK:
            r = g.hierarchize()
        fake.fake_fail(-1)
        assert r in (_lib.SG_OK, _lib.SG_ERR_NOMEM)
        assert fake.sg_set_option(g.h, option, value) == _lib.SG_OK and g.hierarchize() == _lib.SG_OK
        held = g.device_bytes()
        g.close()
        assert fake.fake_live() == start, k
        if r == _lib.SG_OK:
            break
        if k == 0:
            first = held
        assert held == first
        k += 1
    if (d, option) != (3, _lib.SG_OPT_HIER_KERNEL):  # (3, 8) has its chains already
        assert k > 0


def test_options_change_whole_or_not_at_all(fake):
    """A setting whose tables cannot be built is refused and the old one stays,
    under which the grid still works.  The tables' uploads touch neither the
    legacy stream nor a stream that is capturing."""
    g = Grid(fake, 6, 6)
    assert g.set_values() == _lib.SG_OK
    v = C.c_int64()
    for option, value in ((_lib.SG_OPT_HIER_PRECISION, _lib.SG_HIER_FP64), (_lib.SG_OPT_HIER_KERNEL, 2)):
        fake.fake_fail(1)
        assert fake.sg_set_option(g.h, option, value) == _lib.SG_ERR_NOMEM
        assert fake.sg_get_option(g.h, option, C.byref(v)) == _lib.SG_OK and v.value == 0
        allocs = fake.fake_allocs()
        assert fake.sg_hierarchize_async(g.h, None) == _lib.SG_OK and fake.fake_allocs() == allocs
    legacy, unsafe = fake.fake_legacy(), fake.fake_unsafe()
    fake.fake_capture(12345)
    try:
        for option, value in ((_lib.SG_OPT_HIER_PRECISION, _lib.SG_HIER_FP64), (_lib.SG_OPT_HIER_KERNEL, 2),
                              (_lib.SG_OPT_HIER_PRECISION, _lib.SG_HIER_FP32), (_lib.SG_OPT_HIER_KERNEL, 0)):
            assert fake.sg_set_option(g.h, option, value) == _lib.SG_OK
    finally:
        fake.fake_capture(None)
    assert (fake.fake_legacy(), fake.fake_unsafe()) == (legacy, unsafe)
    g.close()


def test_timings_are_of_the_latest_call(fake):
    """A call that does not order its points has no ordering time, whatever an
    earlier one had."""
    g = Grid(fake, 6, 9)
    assert g.set_values() == _lib.SG_OK
    assert fake.sg_set_option(g.h, _lib.SG_OPT_PROFILE, 1) == _lib.SG_OK
    x, ms = np.zeros((60_000, 6), np.float32), np.zeros(_lib.SG_NUM_PHASES)
    for m, ordered in ((60_000, True), (10, False), (60_000, True), (1, False)):
        assert fake.sg_evaluate_device(g.h, x.ctypes.data, x.ctypes.data, m, None) == _lib.SG_OK
        assert fake.sg_timings(g.h, ms.ctypes.data) == _lib.SG_OK
        assert (ms[1] >= 0) == ordered and ms[2] >= 0, m
    g.close()


def test_batch_plans_reuse_their_memory(fake):
    """New offsets or buffers make a new plan; beyond the points' own ordering
    buffers it allocates only what it has no room for."""
    dims, levels = np.array([6, 8, 10], np.int32), np.array([9, 7, 7], np.int32)
    start = fake.fake_live()
    b = C.c_void_p()
    assert fake.sg_batch_create(3, dims.ctypes.data, levels.ctypes.data, None, C.byref(b)) == _lib.SG_OK
    off = np.zeros(4, np.int64)
    fake.sg_batch_offsets(b, off.ctypes.data)
    values = np.zeros(off[3], np.float32)
    assert fake.sg_batch_set_values(b, values.ctypes.data) == _lib.SG_OK
    assert fake.sg_batch_set_option(b, _lib.SG_OPT_EVAL_SORT, 0) == _lib.SG_OK
    x = np.zeros(10 * 4000, np.float32)

    def evaluate(counts):
        po = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        before = fake.fake_allocs(), fake.fake_frees()
        assert fake.sg_batch_evaluate_device(b, po.ctypes.data, x.ctypes.data, x.ctypes.data, None) == _lib.SG_OK
        return fake.fake_allocs() - before[0], fake.fake_frees() - before[1]

    evaluate([1000, 900, 800])
    for counts in ([999, 901, 800], [1, 0, 700], [1000, 900, 800]):
        assert evaluate(counts) == (0, 0), counts
    assert evaluate([1500, 1000, 800])[0] > 0
    assert fake.sg_batch_destroy(b) == _lib.SG_OK
    assert fake.fake_live() == start


@pytest.mark.parametrize("sort", [0, 1])
def test_autotune_leaves_an_untimed_setting_alone(fake, sort):
    """Few points are not ordered under either setting, so the tuner has nothing
    to choose from (all timings are equal here) and a later call with many points
    finds the setting that the caller made."""
    g = Grid(fake, 6, 9)
    assert g.set_values() == _lib.SG_OK
    assert fake.sg_set_option(g.h, _lib.SG_OPT_EVAL_SORT, sort) == _lib.SG_OK
    x, ms, v = np.zeros(600, np.float32), np.zeros(_lib.SG_TUNE_TIMINGS), C.c_int64()
    assert fake.sg_autotune(g.h, x.ctypes.data, x.ctypes.data, 100, None, ms.ctypes.data) == _lib.SG_OK
    assert fake.sg_get_option(g.h, _lib.SG_OPT_EVAL_SORT, C.byref(v)) == _lib.SG_OK and v.value == sort
    g.close()


def test_memory_of_shared_sums(fake):
    """A call that shares its sums returns their memory with its last launch, does
    without where there is none, and allocates under capture only what the handle
    keeps."""
    start = fake.fake_live()
    g = Grid(fake, 6, 9)
    assert g.set_values() == _lib.SG_OK
    x = np.zeros((100, 6), np.float32)

    def evaluate(stream=None):
        return fake.sg_evaluate_device(g.h, x.ctypes.data, x.ctypes.data, 100, stream)

    assert evaluate() == _lib.SG_OK and fake.fake_pool_live() == 0
    live, allocs = fake.fake_live(), fake.fake_allocs()
    assert evaluate() == _lib.SG_OK and (fake.fake_live(), fake.fake_allocs()) == (live, allocs + 1)
    fake.fake_fail(0)
    assert evaluate() == _lib.SG_OK and fake.fake_pool_live() == 0
    unsafe = fake.fake_unsafe()
    fake.fake_capture(12345)
    try:
        assert evaluate(12345) == _lib.SG_OK and fake.fake_live() == live + 1
        assert evaluate() == _lib.SG_OK  # beside the capture
        fake.fake_fail(0)
        assert evaluate(12345) == _lib.SG_OK and fake.fake_live() == live + 1
    finally:
        fake.fake_capture(None)
        fake.fake_fail(-1)
    assert fake.fake_unsafe() == unsafe and fake.fake_pool_live() == 0
    g.close()
    assert fake.fake_live() == start
