"""Levels of odd inner sizes, which a host's own grid may have: 5 cells over 3 over 1,
where the coarse cells' children reach the ghost layer.  An array that ends there and one
with a further layer behind, on the same cells, give the same pressures bit for bit (the
former must not take the pass that reads the children's neighbours)."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from tests import cabi

pytestmark = pytest.mark.gpu
INNER = (5, 3, 1)


class Grid:
    """5^3, 3^3 and 1 inner cells; level 0 in an array of `n`^3 cells.  Ghost cells before
    the inner ones copy their neighbour, those behind keep what they hold."""

    def __init__(self, n):
        self.n = [n, 5, 3]

    def grid_desc(self):
        g = A.GridDesc()
        g.n_levels = 2
        for l, inner in enumerate(INNER):
            for a, b, c, d in (("Nx", "i1", "i2", "dx"), ("Ny", "j1", "j2", "dy"), ("Nz", "k1", "k2", "dz")):
                getattr(g, a)[l], getattr(g, b)[l], getattr(g, c)[l], getattr(g, d)[l] = self.n[l], 1, inner, 0.1 * 2 ** l
        return g

    def at(self, l, i, j, k):
        return i + self.n[l] * (j + self.n[l] * k)

    def list(self, kind, l):
        r = range(1, INNER[l] + 1)
        return np.array([self.at(l, i, j, k) for k in r for j in r for i in r], dtype=np.int64)

    def boundary_program(self, l, ft):
        r = range(1, INNER[l] + 1)
        ops = [op for a in r for b in r for op in ((self.at(l, 0, a, b), self.at(l, 1, a, b)),
                                                   (self.at(l, a, 0, b), self.at(l, a, 1, b)),
                                                   (self.at(l, a, b, 0), self.at(l, a, b, 1)))]
        prog = (A.BcAssign * len(ops))(*[A.BcAssign(target=t, source=s, sign=1, value=0.0) for t, s in ops])
        return np.frombuffer(prog, dtype=A.BC_DTYPE).copy()


@pytest.mark.parametrize("relax", [1, 2])
def test_same_pressure(relax):
    rng = np.random.default_rng(relax)
    p0, rhs = rng.uniform(-1, 1, (2, 7, 7, 7))
    out = []
    for n in (7, 8):
        ctx = cabi.Context(Grid(n))
        try:
            cfg = A.MgCfg(2, 2, 100, relax, 1e-7, 0, 0, 9, 1e-300, 0.6666666667)
            mg, st = C.c_void_p(), A.MgStats()
            A.cuda_check(ctx.lib.artss_mg_create(ctx.h, C.byref(cfg), C.byref(mg)), "mg")
            fields = []
            for f in (p0, rhs):
                big = np.full((n, n, n), 1e6)
                big[:7, :7, :7] = f
                fields.append(ctx.field(big.ravel()))
            for _ in range(3):
                A.cuda_check(ctx.lib.artss_mg_pressure(mg, *fields, 0, C.byref(st)), "pressure")
            out.append(ctx.download(fields[0]).reshape(n, n, n)[:7, :7, :7])
            ctx.lib.artss_mg_destroy(mg)
        finally:
            ctx.close()
    assert np.isfinite(out[0]).all() and np.abs(out[0] - p0).max() > 1e-3
    assert np.array_equal(*out)
