"""axpy_norm's result field: a half field cannot take a full result (refused before any launch), and every other
pairing gives numpy's values."""
import numpy as np
import pytest

import grid_gb300 as g
from tests._common import fermion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(g.F64, 1e-14), (g.F32, 1e-6)])
def test_axpy_norm_shapes(gpu_available, prec, tol):
    dims, Ls = (4, 4, 4, 4), 4
    op = g.MobiusFermion(g.random_gauge(dims, 0.5, 1), dims, Ls, 0.1, 1.8, 1.5, 0.5, precision=prec)
    full, half = [fermion(256, Ls, s) for s in (2, 3)], [fermion(128, Ls, s) for s in (4, 5)]
    fx, fy = (op.FermionField().import_(v) for v in full)
    hx, hy = (op.FermionRedBlackField(g.ODD).import_(v) for v in half)
    with pytest.raises(g.GridError):
        g.axpy_norm(op.FermionRedBlackField(g.ODD), 0.7, fx, fy)
    for x, y, z, (a, b) in ((fx, fy, op.FermionField(), full), (hx, hy, op.FermionRedBlackField(g.ODD), half)):
        want = 0.7 * a + b
        assert abs(g.axpy_norm(z, 0.7, x, y)[0] / np.vdot(want, want).real - 1) < tol
        assert np.linalg.norm(z.export() - want) < tol * np.linalg.norm(want)
