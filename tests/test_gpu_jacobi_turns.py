"""Jacobi diffusion whose arrays take turns (a closed box) and whose input follows
by a copy (a channel with a cube), after odd and even numbers of iterations, both
arrays bit for bit against the oracle, eagerly and in a captured loop."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi, oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.available(), reason="oracle not built")]
P = oracle.p


@pytest.mark.parametrize("scene", ["box", "channel"])
@pytest.mark.parametrize("turbulent", [False, True])
def test_both_arrays(tmp_path, scene, turbulent):
    sc = scenes.channel_with_cube(nx=32, ny=16, nz=16, steps=1, n_level=1) if scene == "channel" else \
        scenes.Scene(nx=33, ny=21, nz=10, X=(0.0, 1.32), Y=(0.0, 0.84), Z=(0.0, 0.4), n_level=0,
                     boundaries=scenes.closed_box_bcs())
    geom = A.Geometry(scenes.write(sc, str(tmp_path / "s.xml")))
    ctx, osc = cabi.Context(geom), oracle.OracleScene(geom)
    lib = ctx.lib
    lib.artss_graph_begin.argtypes = [C.c_void_p]
    lib.artss_graph_end.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_void_p)]
    lib.artss_graph_launch.argtypes = lib.artss_graph_destroy.argtypes = [C.c_void_p]
    try:
        n = ctx.size()
        for captured in (False, True):
            for its in (1, 2, 5, 8, 3):
                rng = np.random.default_rng(its)
                out, inn, b, ev = (rng.uniform(290, 300, n) for _ in range(4))
                ev = 1e-3 * (ev - 290)
                do, di, db, de = (ctx.field(a) for a in (out, inn, b, ev))
                cfg, st, graph = A.IterCfg(its, 1e-300, 1.0), A.IterStats(), C.c_void_p()
                if captured:
                    A.cuda_check(lib.artss_graph_begin(ctx.h), "begin")
                A.cuda_check(lib.artss_diffuse_jacobi(ctx.h, do, di, db, 4.2e-5, de if turbulent else None, 0.01, 5,
                                                      C.byref(cfg), C.byref(st)), "jacobi")
                if captured:
                    A.cuda_check(lib.artss_graph_end(ctx.h, 0, C.byref(graph)), "end")
                    A.cuda_check(lib.artss_graph_launch(graph), "launch")
                res = C.c_double()
                ref = oracle.lib().oracle_diffuse_jacobi(osc.ptr, P(out), P(inn), P(b), 4.2e-5,
                                                         P(ev) if turbulent else None, 0.01, 5, its, 1e-300, 1.0,
                                                         C.byref(res))
                assert ref <= its and (captured or st.iterations == ref)
                assert np.array_equal(ctx.download(do), out)
                assert np.array_equal(ctx.download(di), inn)
                if captured:
                    lib.artss_graph_destroy(graph)
    finally:
        ctx.close()
