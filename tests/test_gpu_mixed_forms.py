"""Mixed-precision cycles with the boundary cells written by the sweeps and the
residual restricted as it is formed, two cells per thread, against the same cycles with
every program launched, the residual stored and one cell per thread (MIXED_BC_LAUNCH): the same pressure, bit for bit
with its boundary cells.  Obstacles apart, touching and none, coarsest levels of a few
cells, pressure conditions with and without values."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import scenes
from tests import cabi

pytestmark = pytest.mark.gpu


def with_outflow(sc, value):
    """the channel's outflow pressure set to `value`"""
    bcs = [(f, p, t, value if f == "p" and t == "dirichlet" else v) for f, p, t, v in sc.boundaries]
    assert any(f == "p" and t == "dirichlet" for f, p, t, v in bcs)
    return dataclasses.replace(sc, boundaries=bcs)


def unaligned(seed):
    boxes = scenes.random_boxes((24, 24, 24), 3, 7, 2, seed, (1.0, 1.0, 1.0), levels=0)
    return scenes.poisson_boxes(n=24, seed=seed, n_level=3, obstacles=boxes)


CASES = {
    "boxes24": lambda: scenes.poisson_boxes(n=24, seed=1, n_level=3),
    "boxes40": lambda: scenes.poisson_boxes(n=40, seed=4, n_level=4),
    "empty16": lambda: scenes.poisson_boxes(n=16, seed=0, n_level=3, obstacles=[], obstacle_bcs=[]),
    "flat": lambda: scenes.poisson_boxes(n=16, seed=0, n_level=2, obstacles=[], obstacle_bcs=[], ny=4, Y=(0.0, 4.0)),
    "channel": lambda: scenes.channel_with_cube(nx=64, ny=32, nz=32, steps=1, n_level=3),
    "channel_valued": lambda: with_outflow(scenes.channel_with_cube(nx=64, ny=32, nz=32, steps=1, n_level=3), 0.25),
    "layered": lambda: scenes.layered_channel(n_level=3),
    "inset": lambda: scenes.inset_box(),
    # obstacles off the coarse cells' edges, odd rows on the finest and on a coarser level
    "unaligned0": lambda: unaligned(0),
    "unaligned3": lambda: unaligned(3),
    "odd15": lambda: scenes.poisson_boxes(n=15, seed=0, n_level=2, obstacles=[], obstacle_bcs=[]),
    "odd18": lambda: scenes.poisson_boxes(n=18, seed=0, n_level=3, obstacles=[], obstacle_bcs=[]),
    "room": lambda: scenes.room_with_door(n=32, n_level=2),
}


@pytest.mark.parametrize("relax", [1, 2, 3])
@pytest.mark.parametrize("case", list(CASES))
def test_forms_agree(case, relax, tmp_path):
    sc = CASES[case]()
    geom = A.Geometry(scenes.write(sc, str(tmp_path / "s.xml")))
    ctx = cabi.Context(geom)
    try:
        rng = np.random.default_rng(relax)
        inner = geom.list("inner", 0)
        p0, b = rng.uniform(-1, 1, ctx.size()), scenes.poisson_rhs(inner, ctx.size(), 3)
        got = []
        for flags in (0, A.MIXED_BC_LAUNCH):
            # three cycles, no tolerance
            cfg = A.MixedCfg(sc.n_level, relax, 1, flags, 0.6666666667, 0.0, 1e-3, 20, 0.0, 3)
            mx = C.c_void_p()
            A.cuda_check(ctx.lib.artss_mixed_create(ctx.h, C.byref(cfg), C.byref(mx)), "mixed")
            dp, db, st = ctx.field(p0), ctx.field(b), A.SolveStats()
            A.cuda_check(ctx.lib.artss_mixed_solve(mx, dp, db, C.byref(st)), "solve")
            ctx.lib.artss_mixed_destroy(mx)
            got.append((st.cycles, st.rel_residual, ctx.download(dp)))
        # the residual's sum over the cells is taken in another order
        assert got[0][0] == got[1][0] and abs(got[0][1] - got[1][1]) <= 1e-12 * got[1][1]
        assert np.array_equal(got[0][2], got[1][2])
        assert not np.array_equal(got[0][2], p0)
    finally:
        ctx.close()
