"""The colored Gauss-Seidel sweep on blocks of 32 x 8 x 4 cells: edges of blocks,
one cell past them, grids smaller than one, both parities of the pitch, obstacles, more
tiles (8400) than a launch has blocks (8192), bit for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi, oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.available(), reason="oracle not built")]
P = oracle.p


@pytest.mark.parametrize("turbulent", [False, True])
@pytest.mark.parametrize("dims", [(32, 8, 4), (33, 9, 5), (64, 16, 8), (3, 3, 3), (31, 7, 13), (95, 41, 22), (33, 9, 8400)])
def test_blocks(tmp_path, dims, turbulent):
    nx, ny, nz = dims
    sc = scenes.Scene(nx=nx, ny=ny, nz=nz, X=(0.0, 0.1 * nx), Y=(0.0, 0.1 * ny), Z=(0.0, 0.1 * nz), steps=1, n_level=0,
                      boundaries=scenes.closed_box_bcs())
    if nx > 90:
        sc.obstacles = [scenes.Box(2.9, 3.5, 0.7, 1.0, 0.3, 1.0, "block")]
        sc.obstacle_bcs = scenes.solid_obstacle_bcs()
    geom = A.Geometry(scenes.write(sc, str(tmp_path / "s.xml")))
    ctx, osc = cabi.Context(geom), oracle.OracleScene(geom)
    try:
        n = ctx.size()
        A.cuda_check(ctx.lib.artss_ctx_sweep_variant(ctx.h, 9), "variant")
        for its in (1, 4):
            rng = np.random.default_rng(its)
            out, inn, b, ev = (rng.uniform(290, 300, n) for _ in range(4))
            ev = 1e-3 * (ev - 290)
            do, di, db, de = (ctx.field(a) for a in (out, inn, b, ev))
            cfg, st, res = A.IterCfg(its, 1e-300, 1.0), A.IterStats(), C.c_double()
            A.cuda_check(ctx.lib.artss_diffuse_cgs(ctx.h, do, di, db, 4.2e-5, de if turbulent else None, 0.01, 5,
                                                   C.byref(cfg), 0, C.byref(st)), "cgs")
            oracle.lib().oracle_diffuse_cgs(osc.ptr, P(out), P(inn), P(b), 4.2e-5, P(ev) if turbulent else None, 0.01, 5,
                                            its, 1e-300, 1.0, C.byref(res))
            assert st.iterations == its and abs(st.residual - res.value) <= 1e-12 * res.value
            assert np.array_equal(ctx.download(do), out)
            assert np.array_equal(ctx.download(di), inn)
    finally:
        ctx.close()
