"""Semi-Lagrangian advection with velocities far outside the grid: the
departure index is clamped to the computational domain on both sides, also
where the displacement in cells exceeds the 32-bit range (a flow that runs
away), so every read stays inside the array."""
import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi

pytestmark = pytest.mark.gpu


def axis(Cn, c, lo, hi):
    """SLAdvect.cpp:79-126 for one axis in unbounded integers."""
    n = np.trunc(Cn)
    pos, neg = Cn > 1e-6, Cn < -1e-6
    c0 = np.where(pos, np.maximum(c - n, lo), np.where(neg, np.minimum(c - n, hi), c))
    c1 = np.where(pos, c0 - 1, np.where(neg, c0 + 1, c))
    return c0.astype(np.int64), c1.astype(np.int64), np.where(pos | neg, np.fmod(np.abs(Cn), 1.0), 1.0)


@pytest.mark.parametrize("speed", [1.0, 3e8, 1e12, 1e300])
def test_runaway_velocity_stays_in_range(tmp_path, speed):
    geom = A.Geometry(scenes.write(scenes.plume_box(n=8, steps=1, n_level=1), str(tmp_path / "box.xml")))
    ctx = cabi.Context(geom)
    try:
        g = ctx.grid
        nx, ny, nz = g.Nx[0], g.Ny[0], g.Nz[0]
        rng = np.random.default_rng(3)
        n = ctx.size()
        vel = [rng.uniform(-speed, speed, n) for _ in range(3)]
        src = rng.standard_normal(n)
        dt = 0.005
        do, ds = ctx.field(np.zeros(n)), ctx.field(src)
        du, dv, dw = (ctx.field(x) for x in vel)
        A.cuda_check(ctx.lib.artss_advect_sl(ctx.h, do, ds, du, dv, dw, dt, A.FIELD_TYPES["T"]), "advect")
        got = ctx.download(do)
        q = geom.list("inner", 0)
        i, j, k = q % nx, q // nx % ny, q // (nx * ny)
        i0, i1, r = axis(dt / g.dx[0] * vel[0][q], i, g.i1[0], g.i2[0])
        j0, j1, s = axis(dt / g.dy[0] * vel[1][q], j, g.j1[0], g.j2[0])
        k0, k1, t = axis(dt / g.dz[0] * vel[2][q], k, g.k1[0], g.k2[0])
        at = lambda a, b, c: src[a + nx * (b + ny * c)]  # noqa: E731
        mix = lambda x, y, w: x + w * (y - x)  # noqa: E731
        want = mix(mix(mix(at(i0, j0, k0), at(i1, j0, k0), r), mix(at(i0, j1, k0), at(i1, j1, k0), r), s),
                   mix(mix(at(i0, j0, k1), at(i1, j0, k1), r), mix(at(i0, j1, k1), at(i1, j1, k1), r), s), t)
        assert np.array_equal(got[q], want)
    finally:
        ctx.close()
