"""Admission of propagator solves (dry run) by the memory that they need, not by the optional fixed-point copies
of their FP64 operator, which a request takes where the budget has room for them."""
import numpy as np
import pytest

import grid_gb300 as g


@pytest.mark.parametrize("dims,Ls,nsrc", [((8, 8, 8, 8), 8, 1), ((16, 8, 4, 8), 12, 4)])
def test_a_request_is_admitted_in_the_memory_it_needs(dims, Ls, nsrc):
    vol = int(np.prod(dims))
    n5 = vol // 2 * Ls * nsrc  # Ls is even: no padding slot
    need = vol * (1152 + 576 + 64 + 576) + n5 * (26 * 192 + 12 * 96)  # links, neighbours, staging; work fields
    copies = vol * 1152 + n5 * 2 * 196
    r = g.make_request(dims, Ls, 0.01, 0.5, 1, nsrc, 2, dry_seconds=0.01)
    assert g.request_bytes(r) == need
    for budget, used in ((need, need), (need + copies - 1, need), (need + copies, need + copies)):
        s = g.Server(budget, slots=1, flags=g.Server.DRY_RUN)
        s.submit(r)
        assert s.wait(1, 10)
        (res,) = s.results()
        assert res.status == 0 and res.chunk == nsrc
        assert s.stats().peak_used_bytes == used
        s.close()
