"""Every compiled mapping of the package's updates: each problem, patch size and precision, with the
method that has compile-time variants (second order, MC limiter) and one that has not.

FP64: bit for bit the CPU oracle's q and CFL numbers.  FP32-wave: relative L1 error of field 0
against the oracle after two steps below 2e-5 (some 150 FP32 roundings of 6e-8 for each step).
Euler's updates that start Newton from the network: the FP64 mappings bit for bit one another (the
same operations in the same order, built without contraction).
"""
import numpy as np
import pytest

from tests.cases import DAM, SHOCKBUBBLE, SPHERE, SWIRL, TSUNAMI, make

pytestmark = pytest.mark.gpu

PROBLEMS = [(DAM, 8), (DAM, 16), (TSUNAMI, 8), (TSUNAMI, 16), (SHOCKBUBBLE, 8), (SHOCKBUBBLE, 16), (SWIRL, 8),
            (SWIRL, 16), (SWIRL, 32), (SPHERE, 8), (SPHERE, 16), (SPHERE, 32)]
IDS = ["dam8", "dam16", "tsunami8", "tsunami16", "bubble8", "bubble16", "swirl8", "swirl16", "swirl32", "sphere8",
       "sphere16", "sphere32"]


def _dt(problem, mx):
    return {8: 0.02, 16: 0.01, 32: 0.005}[mx] * (0.2 if problem in (SPHERE, SHOCKBUBBLE) else 1.0)


def _run(sim, dt):
    return [sim.advance(0.0, dt), sim.advance(dt, dt)], sim.get_q()


def _variants(gc, precision, prepare=lambda g: None):
    """(index, solver) of every variant of a shape, each on a fresh solver."""
    import forestclaw_b200 as fb
    gc.precision = precision
    n = None
    v = 0
    while n is None or v < n:
        g = fb.Solver(gc)
        g.initialize()
        prepare(g)
        n = len(g.variants())
        g.set_variant(v)
        yield v, g
        g.close()
        v += 1


@pytest.mark.parametrize("limiter", [4, 3])
@pytest.mark.parametrize("problem,mx", PROBLEMS, ids=IDS)
def test_every_variant(problem, mx, limiter):
    from oracle import pyoracle as po
    import forestclaw_b200 as fb
    sync = int(problem not in (SWIRL, SPHERE))
    oc, gc = make(problem, mx=mx, my=mx, minlevel=1, maxlevel=2, subcycle=1, time_sync=sync, order=(2, 2),
                  mthlim=(limiter,) * problem["mwaves"])
    o = po.OracleSim(oc)
    o.initialize()
    cfl, q = _run(o, _dt(problem, mx))
    for v, g in _variants(gc, fb.PREC_FP64):
        gcfl, gq = _run(g, _dt(problem, mx))
        assert gcfl == cfl and np.array_equal(gq, q), v
    if problem is SWIRL and mx == 8:
        return                                  # no FP32-wave form of this shape
    inner = (slice(None), 0, slice(2, -2), slice(2, -2))
    for v, g in _variants(gc, fb.PREC_FP32WAVE):
        _, gq = _run(g, _dt(problem, mx))
        assert np.abs(gq[inner] - q[inner]).sum() <= 2e-5 * np.abs(q[inner]).sum(), v


@pytest.mark.parametrize("limiter", [4, 3])
@pytest.mark.parametrize("mx", [8, 16])
def test_every_seeded_variant(mx, limiter):
    import forestclaw_b200 as fb
    _, gc = make(SHOCKBUBBLE, mx=mx, my=mx, minlevel=1, maxlevel=2, subcycle=1, time_sync=1, order=(2, 2),
                 mthlim=(limiter,) * 3)
    m = fb.PStarMLP(seed=0)
    seed = lambda g: g.set_pstar_seed(m)  # noqa: E731
    ref = None
    for v, g in _variants(gc, fb.PREC_FP64, seed):
        got = _run(g, _dt(SHOCKBUBBLE, mx))
        ref = ref or got
        assert got[0] == ref[0] and np.array_equal(got[1], ref[1]), v
    inner = (slice(None), 0, slice(2, -2), slice(2, -2))
    for v, g in _variants(gc, fb.PREC_FP32WAVE, seed):
        _, gq = _run(g, _dt(SHOCKBUBBLE, mx))
        assert np.abs(gq[inner] - ref[1][inner]).sum() <= 2e-5 * np.abs(ref[1][inner]).sum(), v
    m.close()
