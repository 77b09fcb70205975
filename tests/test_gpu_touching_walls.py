"""Boundary programs of several waves (obstacles that touch: the room with a
door) as one launch on the values from before them, bit for bit against the
oracle's sequential loops, and the coarse solves on them in their several forms,
stopped after an odd, an even and the full number of sweeps and by the tolerance."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi, oracle

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not oracle.available(), reason="oracle not built")]
P = oracle.p


@pytest.fixture(scope="module", params=[32, 64])
def room(request, tmp_path_factory):
    geom = A.Geometry(scenes.write(scenes.room_with_door(n=request.param, n_level=2),
                                   str(tmp_path_factory.mktemp("r") / "room.xml")))
    ctx = cabi.Context(geom)
    yield geom, ctx, oracle.OracleScene(geom)
    ctx.close()


def test_programs(room):
    geom, ctx, osc = room
    waves = [ctx.lib.artss_boundary_program_waves(ctx.h, 0, ft) for ft in range(1, 7)]
    assert max(waves) > 1  # the walls touch
    for level in range(geom.levels + 1):
        for ft in range(1, 7):
            if geom.boundary_program(level, ft).size == 0:
                continue
            x = np.random.default_rng(10 * level + ft).uniform(-1, 1, ctx.size(level))
            x[::7] = 0.0
            x[::11] = -0.0
            d = ctx.field(x, level)
            for _ in range(2):
                launches = ctx.lib.artss_ctx_kernel_launches(ctx.h)
                A.cuda_check(ctx.lib.artss_apply_boundary(ctx.h, d, level, ft), "bc")
                assert ctx.lib.artss_ctx_kernel_launches(ctx.h) == launches + 1  # the flat form
                oracle.lib().oracle_apply_bc(osc.ptr, P(x), level, ft)
                got = ctx.download(d, level)
                assert np.array_equal(got, x) and np.array_equal(np.signbit(got), np.signbit(x)), (level, ft)


def pressures(ctx, p0, rhs, sweeps, tol, flags):
    cfg = A.MgCfg(2, 2, 100, 4, 1e-7, 0, flags, sweeps, tol, 0.6666666667)
    mg = C.c_void_p()
    A.cuda_check(ctx.lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(mg)), "mg")
    dp, dr, st, out = ctx.field(p0), ctx.field(rhs), A.MgStats(), []
    for _ in range(3):
        A.cuda_check(ctx.lib.artss_mg_pressure(mg, dp, dr, 0, C.byref(st)), "pressure")
        out.append(ctx.download(dp))
    ctx.lib.artss_mg_destroy(mg)
    return out


@pytest.mark.parametrize("sweeps,tol", [(1, 1e-300), (2, 1e-300), (7, 1e-300), (100, 1e-300), (100, 3.0)])
def test_coarse_solve_forms(room, sweeps, tol):
    """the pipelined coarse solve on the flat program, the cluster and the one-block
    ones on the waves: the same pressure"""
    geom, ctx, osc = room
    rng = np.random.default_rng(sweeps)
    p0, rhs = rng.uniform(-1, 1, ctx.size()), np.zeros(ctx.size())
    inner = geom.list("inner", 0)
    rhs[inner] = rng.uniform(-1, 1, inner.size)
    want = pressures(ctx, p0, rhs, sweeps, tol, 2)
    for flags in (0, 4):
        for a, b in zip(pressures(ctx, p0, rhs, sweeps, tol, flags), want):
            assert np.array_equal(a, b)
