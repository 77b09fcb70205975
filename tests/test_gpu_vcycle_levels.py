"""V-cycles of 1 to 3 levels and 1 to 4 relaxations, on a closed box (every level
takes the short way), a box whose pressure is given on one side (level 0 has a
boundary value, the others do not) and a box with a block that does not line up with
the coarse cells, bit for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi, oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.available(), reason="oracle not built")]
P = oracle.p


def scene(kind):
    bcs = scenes.closed_box_bcs()
    if kind == "given":
        bcs = [bcs[0], ("p", "front,back,bottom,top,left", "neumann", 0.0), ("p", "right", "dirichlet", 0.7), bcs[2]]
    sc = scenes.Scene(nx=32, ny=16, nz=24, X=(0.0, 1.2), Y=(0.0, 0.6), Z=(0.0, 0.9), n_level=3, boundaries=bcs)
    if kind == "block":
        sc.obstacles = [scenes.Box(0.3, 0.6, 0.3, 0.6, 0.3, 0.6, "block")]
        sc.obstacle_bcs = scenes.solid_obstacle_bcs()
    return sc


@pytest.mark.parametrize("kind", ["box", "given", "block"])
def test_pressure(tmp_path, kind):
    geom = A.Geometry(scenes.write(scene(kind), str(tmp_path / "s.xml")))
    ctx, osc = cabi.Context(geom), oracle.OracleScene(geom)
    try:
        n = ctx.size()
        inner = geom.list("inner", 0)
        for levels in (1, 2, 3):
            for relax in (1, 2, 3, 4):
                rng = np.random.default_rng(levels + 10 * relax)
                p0, rhs = rng.uniform(-1, 1, n), np.zeros(n)
                rhs[inner] = rng.uniform(-1, 1, inner.size)
                cycles = 1 + relax % 2
                cfg = A.MgCfg(levels, cycles, 100, relax, 1e-7, 0, 0, 9, 1e-300, 0.6666666667)
                ocfg = oracle.MgCfg(levels, cycles, 100, relax, 1e-7, 0, 0, 9, 1e-300, 0.6666666667)
                mg, om = C.c_void_p(), oracle.lib().oracle_mg_create(osc.ptr, C.byref(ocfg))
                A.cuda_check(ctx.lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(mg)), "mg")
                dp, dr, st, res = ctx.field(p0), ctx.field(rhs), A.MgStats(), C.c_double()
                for _ in range(2):
                    A.cuda_check(ctx.lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
                    oracle.lib().oracle_mg_pressure(om, P(p0), P(rhs), 0, C.byref(res))
                    assert np.array_equal(ctx.download(dp), p0), (levels, relax)
                ctx.lib.artss_mg_destroy(mg)
                oracle.lib().oracle_mg_destroy(om)
    finally:
        ctx.close()
