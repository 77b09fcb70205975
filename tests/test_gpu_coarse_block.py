"""The one-block Jacobi coarse solve of small levels against the cluster and the older
one-block forms: the same pressures bit for bit, stopped after one to all sweeps and by
the tolerance, for programs of one wave, flat ones, valued ones and levels of one and of
two cells per thread."""
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
