"""The one-block Jacobi coarse solve of small levels against the cluster and the older
one-block forms: the same pressures bit for bit, stopped after one to all sweeps and by
the tolerance, for programs of one wave, flat ones, valued ones and levels of one and of
two cells per thread."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi
from tests.test_gpu_touching_walls import pressures

pytestmark = pytest.mark.gpu


def outflow(value):
    sc = scenes.channel_with_cube(nx=32, ny=16, nz=16, steps=1, n_level=2)
    sc.boundaries = [(f, p, t, value if f == "p" and t == "dirichlet" else v) for f, p, t, v in sc.boundaries]
    return sc


SCENES = {
    "cube4": lambda: scenes.plume_box(n=8, n_level=2),
    "cube8": lambda: scenes.plume_box(n=16, n_level=2),
    "cube9": lambda: scenes.plume_box(n=18, n_level=2),
    "cube11": lambda: scenes.plume_box(n=22, n_level=2),
    "room": lambda: scenes.room_with_door(n=16, n_level=2),
    "channel": lambda: outflow(0.0),
    "channel_valued": lambda: outflow(0.25),
}


@pytest.mark.parametrize("name", list(SCENES))
def test_forms(name, tmp_path):
    geom = A.Geometry(scenes.write(SCENES[name](), str(tmp_path / "s.xml")))
    ctx = cabi.Context(geom)
    try:
        inner = geom.list("inner", 0)
        for sweeps, tol in [(1, 1e-300), (2, 1e-300), (3, 1e-300), (4, 1e-300), (7, 1e-300), (100, 1e-300), (100, 3.0)]:
            rng = np.random.default_rng(sweeps)
            p0, rhs = rng.uniform(-1, 1, ctx.size()), np.zeros(ctx.size())
            rhs[inner] = rng.uniform(-1, 1, inner.size)
            got = pressures(ctx, p0, rhs, sweeps, tol, 0)
            for flags in (2, 4):
                for a, b in zip(pressures(ctx, p0, rhs, sweeps, tol, flags), got):
                    assert np.array_equal(a, b), (sweeps, tol, flags)
    finally:
        ctx.close()


@pytest.mark.parametrize("chain", [False, True])
def test_assigned_inner_cells(tmp_path, chain):
    """A program that also assigns inner cells of the coarse solve's level, from a cell that
    nothing writes and (chain: a flat program) from one another: the other forms' bits."""
    geom = A.Geometry(scenes.write(SCENES["cube8"](), str(tmp_path / "s.xml")))
    ctx = cabi.Context(geom)
    try:
        prog = geom.boundary_program(1, 4)
        prog = np.ascontiguousarray(prog[(prog["target"] != 0) & (prog["source"] != 0)])  # nothing writes the array's first cell
        nx, nxy = ctx.grid.Nx[1], ctx.grid.Nx[1] * ctx.grid.Ny[1]
        at = lambda i, j, k: i + nx * j + nxy * k  # noqa: E731
        # (target, source): inner from a constant cell, inner from inner
        more = [(at(4, 4, 4), at(0, 0, 0)), (at(5, 2, 6), at(3, 3, 3))]
        if chain:  # a cell that is read before it is written: several waves
            more = [(at(6, 6, 6), at(4, 4, 4))] + more
        arr = (A.BcAssign * (prog.size + len(more)))()
        C.memmove(arr, prog.ctypes.data, prog.nbytes)
        for n, (t, s) in enumerate(more):
            arr[prog.size + n] = A.BcAssign(target=t, source=s, sign=1, value=0.25)
        A.cuda_check(ctx.lib.artss_set_boundary_program(ctx.h, 1, 4, arr, prog.size + len(more)), "bc")
        assert (ctx.lib.artss_boundary_program_waves(ctx.h, 1, 4) > 1) == chain
        inner = geom.list("inner", 0)
        for sweeps in (1, 2, 3, 20):
            rng = np.random.default_rng(sweeps)
            p0, rhs = rng.uniform(-1, 1, ctx.size()), np.zeros(ctx.size())
            rhs[inner] = rng.uniform(-1, 1, inner.size)
            got = pressures(ctx, p0, rhs, sweeps, 1e-300, 0)
            for flags in (2, 4):
                for a, b in zip(pressures(ctx, p0, rhs, sweeps, 1e-300, flags), got):
                    assert np.array_equal(a, b), (sweeps, flags)
    finally:
        ctx.close()
