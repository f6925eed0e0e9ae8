"""fc2d_b200_restore_step returns once q is restored: nothing is left on the solver's stream."""
import numpy as np
import pytest

from tests.cases import DAM, make

pytestmark = pytest.mark.gpu


def test_restore_step_leaves_an_idle_stream():
    import torch
    import forestclaw_b200 as fb
    _, gc = make(DAM, mx=16, my=16, minlevel=6, maxlevel=6)
    g = fb.Solver(gc)
    g.initialize()
    q = g.get_q()
    st = torch.cuda.ExternalStream(g.stream_handle())
    for _ in range(50):                 # 50 copies of 39 MB in stream order: half a millisecond of work
        g.save_step()
    g.restore_step()
    assert st.query()
    assert np.array_equal(g.get_q(), q)
