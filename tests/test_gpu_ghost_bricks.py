"""Ghost fill on bricks of blocks: every ghost cell, bit for bit the CPU oracle's.

A forest of one level fills its neighbours' cells and its physical boundary in one launch, where
a boundary cell beside another patch takes its value from that patch's interior; a refined one
keeps the two apart.  Walls, extrapolation and an inflow side meet at corners of the domain, at
block edges and on forests one patch wide.
"""
import numpy as np
import pytest

from tests.cases import DAM, SHOCKBUBBLE, SWIRL, make

pytestmark = pytest.mark.gpu

BRICKS = [(1, 1, 0, 0), (3, 1, 0, 0), (1, 3, 0, 0), (3, 2, 1, 1), (2, 3, 0, 2)]
PROBLEMS = [(DAM, 8, (3, 1, 1, 3)), (DAM, 16, (3, 3, 3, 3)), (SHOCKBUBBLE, 16, (0, 1, 3, 3)), (SWIRL, 8, (1, 1, 1, 1))]


@pytest.mark.parametrize("mi,mj,minlevel,maxlevel", BRICKS)
@pytest.mark.parametrize("problem,mx,mthbc", PROBLEMS, ids=["dam8", "dam16", "bubble16", "swirl8"])
def test_ghost_cells_of_a_brick(problem, mx, mthbc, mi, mj, minlevel, maxlevel):
    from oracle import pyoracle as po
    import forestclaw_b200 as fb
    sync = int(problem is not SWIRL)
    oc, gc = make(problem, mx=mx, my=mx, mi=mi, mj=mj, minlevel=minlevel, maxlevel=maxlevel, mthbc=mthbc, subcycle=1,
                  time_sync=sync)
    o, g = po.OracleSim(oc), fb.Solver(gc)
    o.initialize()
    g.initialize()
    q0 = o.get_q()
    assert np.array_equal(g.get_q(), q0)
    # a state that no symmetry of the domain maps to itself
    rng = np.random.default_rng(mi * 10 + mj)
    q0 = q0 * (1.0 + 0.05 * rng.random(q0.shape))
    o.set_q(q0)
    g.set_q(q0)
    t, dt = 0.0, 0.02 / mx
    for _ in range(3):
        assert g.advance(t, dt) == o.advance(t, dt)
        t += dt
    q = o.get_q()
    assert np.isfinite(q).all()
    assert np.array_equal(g.get_q(), q)
