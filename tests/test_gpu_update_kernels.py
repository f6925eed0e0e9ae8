"""The fused update kernels over the methods they accept: order, transverse order and limiter
(one on every wave, fixed at compile time or not, and mixed), patch sizes, walls.

FP64: bit for bit the CPU oracle's q and CFL numbers.  FP32-wave: relative L1 error of field 0
against the oracle after two steps below 2e-5, i.e. some 150 FP32 roundings (6e-8 each, about
the operations behind one flux) for each of the two steps.
"""
import numpy as np
import pytest

from tests.cases import DAM, SHOCKBUBBLE, SPHERE, SWIRL, TSUNAMI, make

pytestmark = pytest.mark.gpu

METHODS = [((2, 2), (4, 4, 4)), ((2, 2), (3, 3, 3)), ((2, 2), (4, 1, 4)), ((2, 1), (2, 2, 2)), ((2, 0), (1, 1, 1)),
           ((1, 1), (4, 4, 4)), ((1, 0), (0, 0, 0)), ((2, 2), (6, 6, 6)), ((2, 2), (0, 0, 0))]
PROBLEMS = [(DAM, 8, dict(mthbc=(3, 3, 3, 3))), (DAM, 16, {}), (TSUNAMI, 8, {}), (TSUNAMI, 16, dict(mthbc=(3, 1, 1, 3))),
            (SHOCKBUBBLE, 8, {}), (SHOCKBUBBLE, 16, {}), (SWIRL, 8, {}), (SWIRL, 16, {}), (SWIRL, 32, {}), (SPHERE, 8, {}),
            (SPHERE, 16, {})]
IDS = ["dam8", "dam16", "tsunami8", "tsunami16", "bubble8", "bubble16", "swirl8", "swirl16", "swirl32", "sphere8", "sphere16"]


def _run(sim, dt):
    cfl, t = [], 0.0
    for _ in range(2):
        cfl.append(sim.advance(t, dt))
        t += dt
    return sim.get_q(), cfl


@pytest.mark.parametrize("order,mthlim", METHODS)
@pytest.mark.parametrize("problem,mx,kw", PROBLEMS, ids=IDS)
def test_update_over_methods(problem, mx, kw, order, mthlim):
    from oracle import pyoracle as po
    import forestclaw_b200 as fb
    sync = int(problem not in (SWIRL, SPHERE))
    kw = dict(kw, mx=mx, my=mx, minlevel=1, maxlevel=2, subcycle=1, time_sync=sync, order=order,
              mthlim=mthlim[:problem["mwaves"]])
    oc, gc = make(problem, **kw)
    o = po.OracleSim(oc)
    o.initialize()
    dt = {8: 0.02, 16: 0.01, 32: 0.005}[mx] * (0.2 if problem in (SPHERE, SHOCKBUBBLE) else 1.0)
    q, cfl = _run(o, dt)
    assert np.isfinite(q).all()
    g = fb.Solver(gc)
    g.initialize()
    gq, gcfl = _run(g, dt)
    assert gcfl == cfl
    assert np.array_equal(gq, q)
    if problem is SWIRL and mx == 8:
        return                                  # no FP32-wave form of this shape
    gc.precision = fb.PREC_FP32WAVE
    g = fb.Solver(gc)
    g.initialize()
    fq, _ = _run(g, dt)
    inner = (slice(None), 0, slice(2, -2), slice(2, -2))
    assert np.abs(fq[inner] - q[inner]).sum() <= 2e-5 * np.abs(q[inner]).sum()
