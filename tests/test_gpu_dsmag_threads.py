"""Dynamic Smagorinsky in contexts of different sizes side by side: calls from two
host threads, and a call of a small grid between the capture of a large one's and the
graph's instantiation.  Their averaging kernels take different amounts of shared memory
(181 KB at 96 rows, 67 KB at 16), whose limit is the function's."""
import ctypes as C
import threading

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi

pytestmark = pytest.mark.gpu


class Member:
    def __init__(self, path, dims):
        nx, ny, nz = dims
        sc = scenes.Scene(nx=nx, ny=ny, nz=nz, X=(0.0, 0.1 * nx), Y=(0.0, 0.1 * ny), Z=(0.0, 0.1 * nz), steps=1, n_level=0,
                          boundaries=scenes.closed_box_bcs())
        self.ctx = cabi.Context(A.Geometry(scenes.write(sc, str(path))))
        rng = np.random.default_rng(ny)
        self.uvw = [self.ctx.field(rng.uniform(-1, 1, self.ctx.size())) for _ in range(3)]
        self.ev = self.ctx.field()
        self.bad = []

    def call(self, times=1):
        for _ in range(times):
            st = self.ctx.lib.artss_turb_dynamic_smagorinsky(self.ctx.h, self.ev, *self.uvw, 1e-3)
            if st:
                self.bad.append(st)

    def result(self):
        return self.ctx.download(self.ev)


@pytest.fixture
def pair(tmp_path):
    members = [Member(tmp_path / "a.xml", (3, 96, 10)), Member(tmp_path / "b.xml", (3, 16, 12))]
    for m in members:
        m.call()
        m.want = m.result()
    yield members
    for m in members:
        m.ctx.close()


def test_two_threads(pair):
    for _ in range(3):
        threads = [threading.Thread(target=m.call, args=(3000,)) for m in pair]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for m in pair:
            assert not m.bad
            assert np.array_equal(m.result(), m.want)


def test_small_call_between_capture_and_instantiation(pair):
    large, small = pair
    lib = large.ctx.lib
    lib.artss_graph_begin.argtypes = [C.c_void_p]
    lib.artss_graph_end.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_void_p)]
    lib.artss_graph_launch.argtypes = lib.artss_graph_destroy.argtypes = [C.c_void_p]
    A.cuda_check(lib.artss_fill(large.ctx.h, large.ev, 0, 0.0), "fill")
    graph = C.c_void_p()
    A.cuda_check(lib.artss_graph_begin(large.ctx.h), "begin")
    large.call()
    small.call()
    A.cuda_check(lib.artss_graph_end(large.ctx.h, 0, C.byref(graph)), "end")
    A.cuda_check(lib.artss_graph_launch(graph), "launch")
    assert not large.bad + small.bad
    for m in pair:
        assert np.array_equal(m.result(), m.want)
    lib.artss_graph_destroy(graph)


def test_a_wait_that_runs_out_is_reported(pair):
    """two blocks of five planes; the second one's wait for the first runs out at once"""
    large, small = pair
    lib, h = large.ctx.lib, large.ctx.h
    A.cuda_check(lib.artss_ctx_wait_limit(h, 0), "limit")
    large.call()
    small.call()
    assert not large.bad and lib.artss_ctx_sync(h) == -2  # ARTSS_ERR_CUDA
    assert "averaging" in lib.artss_last_error().decode()
    assert np.isnan(large.result()).any()  # reported once
    large.call()
    with pytest.raises(RuntimeError):
        large.result()
    A.cuda_check(lib.artss_ctx_wait_limit(h, -1), "limit")
    for m in pair:
        m.call()
        assert lib.artss_ctx_sync(m.ctx.h) == 0 and np.array_equal(m.result(), m.want)
