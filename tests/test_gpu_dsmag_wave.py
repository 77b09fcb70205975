"""Dynamic Smagorinsky on grids where the averaging's blocks hold all planes, a
few each, a part of the last ones, and on rows too many for them (the grid-barrier
form), bit for bit against the oracle's loops."""
import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi, oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.available(), reason="oracle not built")]


@pytest.mark.parametrize("dims,cube", [((16, 16, 16), False), ((37, 19, 5), False), ((24, 130, 11), False),
                                       ((9, 300, 7), False), ((6, 520, 3), False), ((80, 48, 56), True),
                                       ((33, 41, 90), False)])
def test_against_the_loops(tmp_path, dims, cube):
    nx, ny, nz = dims
    sc = scenes.Scene(nx=nx, ny=ny, nz=nz, X=(0.0, 0.1 * nx), Y=(0.0, 0.1 * ny), Z=(0.0, 0.1 * nz), steps=1, n_level=0,
                      boundaries=scenes.closed_box_bcs())
    if cube:
        sc.obstacles = [scenes.Box(1.6, 2.4, 0.8, 2.0, 1.2, 3.0, "cube")]
        sc.obstacle_bcs = scenes.solid_obstacle_bcs()
    geom = A.Geometry(scenes.write(sc, str(tmp_path / "s.xml")))
    ctx, osc = cabi.Context(geom), oracle.OracleScene(geom)
    try:
        n = ctx.size()
        for seed in (1, 2):
            rng = np.random.default_rng(seed)
            u, v, w, ev = (rng.uniform(-1, 1, n) for _ in range(4))
            du, dv, dw, dev = (ctx.field(a) for a in (u, v, w, ev))
            A.cuda_check(ctx.lib.artss_turb_dynamic_smagorinsky(ctx.h, dev, du, dv, dw, 1e-3), "dynamic smagorinsky")
            oracle.lib().oracle_dynamic_smagorinsky(osc.ptr, oracle.p(ev), oracle.p(u), oracle.p(v), oracle.p(w), 1e-3)
            assert np.array_equal(ctx.download(dev), ev)
    finally:
        ctx.close()
