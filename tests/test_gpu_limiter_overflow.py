"""FP32-wave limiter: waves whose squares overflow FP32 are reported, not limited as if in range.

The ratio of the limiter is then inf/inf, so the limited wave is NaN; it must reach q, which the
next step reports.  Everything else stays in range: the same data without a limiter, and the FP64
form, go through both steps.
"""
import numpy as np
import pytest

from tests.cases import DAM, SWIRL, make

pytestmark = pytest.mark.gpu

# steep but smooth fields: field 0 = scale * (2 + i/10) along x.  Dam: h ~ 1e15, so the acoustic
# waves' momentum is some 1e21 (square above 3.4e38), the flux differences below 1e31.
CASES = [(DAM, 8, 1e15, 1e-10), (DAM, 16, 1e15, 1e-10), (SWIRL, 16, 1e21, 1e-3), (SWIRL, 32, 1e21, 1e-3)]


def _two_steps(problem, mx, scale, dt, precision, limiter):
    import forestclaw_b200 as fb
    _, gc = make(problem, mx=mx, my=mx, minlevel=1, maxlevel=1, order=(2, 2), mthlim=(limiter,) * problem["mwaves"])
    gc.precision = precision
    g = fb.Solver(gc)
    g.initialize()
    q = np.zeros_like(g.get_q())
    q[:, 0] = scale * (2.0 + 0.1 * np.arange(q.shape[-1]))
    g.set_q(q)
    g.advance(0.0, dt)
    g.advance(dt, dt)
    return g.get_q()


@pytest.mark.parametrize("problem,mx,scale,dt", CASES, ids=["dam8", "dam16", "swirl16", "swirl32"])
def test_overflowing_limiter_ratio_is_reported(problem, mx, scale, dt):
    import forestclaw_b200 as fb
    assert np.isfinite(_two_steps(problem, mx, scale, dt, fb.PREC_FP64, 4)).all()
    assert np.isfinite(_two_steps(problem, mx, scale, dt, fb.PREC_FP32WAVE, 0)).all()
    with pytest.raises(fb.B200Error, match="non-finite"):
        _two_steps(problem, mx, scale, dt, fb.PREC_FP32WAVE, 4)
