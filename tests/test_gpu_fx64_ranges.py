"""The fixed-point form of the FP64 hopping term (grid_gb300/csrc/gb_dhop_fx.cu) on inputs whose numbers
differ in size inside one block: links.  FP64 arithmetic keeps each of them; the bound is that of
test_gpu_fx64.py (1e-15 per site)."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import fermion
from tests.test_gpu_fx64 import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [20, 3, -8, -30])
@pytest.mark.parametrize("kind,Ls", [("wilson", 1), ("mobius", 8)])
def test_links_of_different_sizes(gpu_available, kind, Ls, power):
    """A few links 2^power of the others: each output is as accurate as its own terms, also where it touches
    no scaled link."""
    dims, vol = (4, 4, 4, 6), 384
    U = g.random_gauge(dims, 0.5, 81).reshape(vol * 4, 9).copy()
    if power > 0:
        U[[5, 700]] *= 2.0 ** power
    else:  # whole neighbourhoods, so that some sums have small terms only
        U[:1200] *= 2.0 ** power
    op, ref = make(kind, dims, Ls, 1, U.reshape(-1))
    x = fermion(vol // 2, Ls, 82)
    for dag in (0, 1):
        fi, fo = op.FermionRedBlackField(g.ODD).import_(x), op.FermionRedBlackField(g.EVEN)
        op.DhopEO(fi, fo, dag)
        got, want = fo.export().reshape(-1, 12), ref.dhop_cb(x, 1, dag).reshape(-1, 12)
        err, size = np.linalg.norm(got - want, axis=1), np.linalg.norm(want, axis=1)
        assert (err <= 1e-15 * size).all(), (dag, (err / size).max())
