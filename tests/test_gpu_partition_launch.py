"""The ghost-fill launches of one rank of a partitioned forest cover what that rank fills.

One solver plays one rank of many (no transport: the exchange does nothing, so values are not
looked at).  A rank far from a small refined region has no ghost cell of the fine level to fill and
launches nothing for it; a rank beside it does.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _NoTransport:
    def __init__(self, rank, size):
        from forestclaw_b200 import partition as pt
        self._keep = (pt.EXCHANGE_FN(lambda *a: 0), pt.REDUCE_FN(lambda *a: 0), pt.REDUCE_FN(lambda *a: 0))
        self.c = pt.Comm(rank, size, None, *self._keep)


def test_rank_without_fine_patches_launches_no_fine_copy():
    import forestclaw_b200 as fb
    from forestclaw_b200 import partition as pt
    from tests.cases import DAM, make
    size = 16
    # level 3 uniform, the patch at the origin refined
    leaves = [(3, x, y) for y in range(8) for x in range(8) if x or y] + [(4, x, y) for y in range(2) for x in range(2)]
    lev, gx, gy = (np.array(v) for v in zip(*leaves))
    _, gc = make(DAM, mx=8, my=8, minlevel=3, maxlevel=4, subcycle=1)

    def launches(rank):
        g = fb.Solver(gc)
        pt.partition(g, _NoTransport(rank, size))
        g.set_forest(lev, gx, gy)
        info, owner = g.patch_info(), g.partition_owner()
        n0 = g.last_update_stats()["total_launches"]
        g.ghost_update(4, 4, 0.0)
        g.synchronize()
        n = g.last_update_stats()["total_launches"] - n0
        fine = set(owner[info[:, 0] == 4])
        g.close()
        return n, fine

    n0, fine = launches(0)
    assert 0 in fine and size - 1 not in fine
    assert n0 > 0
    assert launches(size - 1)[0] == 0
