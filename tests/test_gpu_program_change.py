"""A multigrid solver whose context gets other cell lists and boundary programs after
its creation: from a closed box to a box with a block and touching walls, to a given
pressure, and back.  Each later call, eager, replayed from a graph and relative, gives
the bits of a solver created after the change."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi

pytestmark = pytest.mark.gpu
I64P = C.POINTER(C.c_int64)


def scene(kind):
    bcs = scenes.closed_box_bcs()
    if kind == "given":
        bcs = [bcs[0], ("p", "front,back,bottom,top,left", "neumann", 0.0), ("p", "right", "dirichlet", 0.7), bcs[2]]
    sc = scenes.Scene(nx=32, ny=16, nz=32, X=(0.0, 1.6), Y=(0.0, 0.8), Z=(0.0, 1.6), n_level=3, boundaries=bcs)
    if kind == "walls":
        sc.obstacles = [scenes.Box(0.4, 0.8, 0.4, 0.8, 0.4, 0.8, "block"), scenes.Box(0.8, 1.2, 0.4, 0.8, 0.4, 1.2, "wall"),
                        scenes.Box(0.0, 0.4, 0.0, 0.4, 0.8, 1.2, "corner")]
        sc.obstacle_bcs = scenes.solid_obstacle_bcs()
    return sc


def apply(ctx, geom):
    """the lists and programs of `geom` in a context of the same grid"""
    for level in range(ctx.grid.n_levels + 1):
        lists = [np.ascontiguousarray(geom.list(k, level)) for k in ("inner", "domain")]
        args = [x for v in lists for x in (v.ctypes.data_as(I64P), v.size)]
        A.cuda_check(ctx.lib.artss_set_cell_lists(ctx.h, level, *args), "lists")
        for ft in range(7):
            prog = geom.boundary_program(level, ft)
            arr = (A.BcAssign * max(prog.size, 1))()
            C.memmove(arr, prog.ctypes.data, prog.nbytes)
            A.cuda_check(ctx.lib.artss_set_boundary_program(ctx.h, level, ft, arr, prog.size), "bc")


@pytest.mark.parametrize("relax", [1, 2])
def test_solver_follows(tmp_path, relax):
    geoms = {k: A.Geometry(scenes.write(scene(k), str(tmp_path / f"{k}.xml"))) for k in ("box", "walls", "given")}
    ctx = cabi.Context(geoms["box"])
    lib = ctx.lib
    cfg = A.MgCfg(3, 2, 100, relax, 1e-7, 0, 0, 9, 1e-300, 0.6666666667)
    try:
        old = C.c_void_p()
        A.cuda_check(lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(old)), "mg")
        dp, dr, st, ss = ctx.field(), ctx.field(), A.MgStats(), A.SolveStats()
        for n, kind in enumerate(("box", "walls", "given", "walls", "box")):
            if n:
                apply(ctx, geoms[kind])
            rng = np.random.default_rng(n)
            p0, rhs = rng.uniform(-1, 1, ctx.size()), np.zeros(ctx.size())
            inner = geoms[kind].list("inner", 0)
            rhs[inner] = rng.uniform(-1, 1, inner.size)
            ctx.upload(dr, rhs)
            new = C.c_void_p()
            A.cuda_check(lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(new)), "mg")
            got = []
            for mg in (old, new):
                ctx.upload(dp, p0)
                out = []
                for _ in range(3):
                    A.cuda_check(lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
                    out.append(ctx.download(dp))
                A.cuda_check(lib.artss_mg_set_rhs(mg, dp, dr), "rhs")
                A.cuda_check(lib.artss_mg_vcycle(mg, dp), "cycle")
                out.append(ctx.download(dp))
                A.cuda_check(lib.artss_mg_solve_rel(mg, dp, dr, 0.0, 2, C.byref(ss)), "relative")
                got.append(out + [ctx.download(dp)])
            lib.artss_mg_destroy(new)
            for a, b in zip(*got):
                assert np.isfinite(b).all() and np.array_equal(a, b), (n, kind)
        lib.artss_mg_destroy(old)
    finally:
        ctx.close()


def test_captured_after_a_change(tmp_path):
    """a change, then a capture before any eager call: the replay and the eager calls
    after it give a new solver's bits"""
    geoms = {k: A.Geometry(scenes.write(scene(k), str(tmp_path / f"{k}.xml"))) for k in ("box", "walls")}
    ctx = cabi.Context(geoms["box"])
    lib = ctx.lib
    lib.artss_graph_begin.argtypes = [C.c_void_p]
    lib.artss_graph_end.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_void_p)]
    lib.artss_graph_launch.argtypes = lib.artss_graph_destroy.argtypes = [C.c_void_p]
    cfg = A.MgCfg(3, 2, 100, 2, 1e-7, 0, 0, 9, 1e-300, 0.6666666667)
    try:
        rng = np.random.default_rng(3)
        p0, rhs = rng.uniform(-1, 1, ctx.size()), np.zeros(ctx.size())
        inner = geoms["walls"].list("inner", 0)
        rhs[inner] = rng.uniform(-1, 1, inner.size)
        dp, dr, st, mg, new, graph = ctx.field(p0), ctx.field(rhs), A.MgStats(), C.c_void_p(), C.c_void_p(), C.c_void_p()
        A.cuda_check(lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(mg)), "mg")
        A.cuda_check(lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
        apply(ctx, geoms["walls"])
        A.cuda_check(lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(new)), "mg")
        ctx.upload(dp, p0)
        want = []
        for _ in range(4):
            A.cuda_check(lib.artss_mg_pressure(new, dp, dr, 0, C.byref(st)), "pressure")
            want.append(ctx.download(dp))
        ctx.upload(dp, p0)
        A.cuda_check(lib.artss_graph_begin(ctx.h), "begin")
        A.cuda_check(lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
        A.cuda_check(lib.artss_graph_end(ctx.h, 0, C.byref(graph)), "end")
        for n in range(2):
            A.cuda_check(lib.artss_graph_launch(graph), "launch")
            assert np.array_equal(ctx.download(dp), want[n])
        for n in range(2, 4):
            A.cuda_check(lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
            assert np.array_equal(ctx.download(dp), want[n])
        lib.artss_graph_destroy(graph)
        lib.artss_mg_destroy(mg)
        lib.artss_mg_destroy(new)
    finally:
        ctx.close()
