"""A staging copy that does not arrive: the update reports it and writes nothing else.

tests/user_solvers/stage_lost_user.cu builds the package's kernels so that they take every staging copy
for lost.  q must stay as it was, and so must the values time interpolation starts from
(save_current_step), which show in the ghost cells it fills; no other failure is reported, although
the data, were it looked at, holds a negative depth.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _module():
    import forestclaw_b200 as fb
    from forestclaw_b200 import build
    fb.load_library()
    return ctypes.CDLL(next(p for p in build.build_user_examples() if p.endswith("libstage_lost_user.so")))


def _interpolated(g, q):
    """q after the fine level's ghost cells were filled from the coarse values saved before its
    last step (alpha = 0: the saved values alone)."""
    g.set_q(q)
    g._check("fc2d_b200_timeinterp", g.lib.fc2d_b200_timeinterp(g.h, 1, 0.0))
    g.ghost_update(2, 2, 0.0, 1)
    return g.get_q()


@pytest.mark.parametrize("how,meqn,maux", [("inline", 3, 0), ("advection", 1, 2)])
def test_lost_staging_copy_writes_nothing(how, meqn, maux):
    import forestclaw_b200 as fb
    g = fb.Solver(fb.Options(mx=8, my=8, mbc=2, meqn=meqn, maux=maux, mwaves=3 if meqn == 3 else 1, minlevel=1, maxlevel=2,
                             subcycle=1, time_sync=0, mthbc=(1, 1, 1, 1), rp=fb.RP_USER, app=fb.APP_NONE))
    fn = getattr(_module(), "stage_lost_register_" + how)
    fn.argtypes = [ctypes.c_void_p]
    assert fn(g.h) == 0, g.lib.fc2d_b200_last_error()
    # three coarse patches and four fine ones
    g.set_forest([1, 1, 1, 2, 2, 2, 2], [1, 0, 1, 0, 1, 0, 1], [0, 1, 1, 0, 0, 1, 1])
    rng = np.random.default_rng(1)
    q = rng.uniform(1.0, 2.0, g.get_q().shape)
    saved = _interpolated(g, q)
    bad = q.copy()
    bad[:, 0] -= 1.5                                    # negative in places
    g.set_q(bad)
    with pytest.raises(fb.B200Error) as e:
        g.level_update(1, 0.0, 1e-3)
    assert "did not complete" in str(e.value)
    assert "negative" not in str(e.value) and "non-finite" not in str(e.value)
    assert np.array_equal(g.get_q(), bad)
    assert np.array_equal(_interpolated(g, q), saved, equal_nan=True)
    g.close()
