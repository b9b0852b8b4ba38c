"""The force kernel at its edges: sites that do not fill a warp, a single vector along s (one lane
per site), uneven walks of the two lanes, several right-hand sides with a padding slot.  FP64
relative L2 1e-13, FP32 1e-6, as the operators' parity bounds."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import MOBIUS, fermion

pytestmark = pytest.mark.gpu

TOL = {g.F64: 1e-13, g.F32: 1e-6}


@pytest.mark.parametrize("prec", [g.F64, g.F32])
@pytest.mark.parametrize("kind,dims,Ls,nrhs", [("wilson", (2, 2, 2, 2), 1, 1), ("wilson", (2, 2, 6, 2), 1, 3),
                                               ("wilson", (4, 2, 2, 10), 1, 4), ("mobius", (2, 2, 2, 6), 2, 1),
                                               ("mobius", (4, 2, 6, 6), 10, 1), ("mobius", (2, 4, 2, 2), 6, 3)])
def test_force_edges(gpu_available, prec, kind, dims, Ls, nrhs):
    U, ph, vol = g.random_gauge(dims, 0.5, 51), g.antiperiodic_t(), int(np.prod(dims))
    if kind == "wilson":
        op = g.WilsonFermion(U, dims, 0.1, precision=prec, nrhs=nrhs)
        ref = o.OracleOp(0, 0, dims, 1, [0.1], U, ph)
    else:
        par = [0.05, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
        op = g.MobiusFermion(U, dims, Ls, *par, precision=prec, nrhs=nrhs)
        ref = o.OracleOp(1, 0, dims, Ls, par, U, ph)
    A, B = fermion(vol * nrhs, Ls, 52).reshape(nrhs, -1), fermion(vol * nrhs, Ls, 53).reshape(nrhs, -1)
    fa, fb = op.FermionField().import_(A.reshape(-1)), op.FermionField().import_(B.reshape(-1))
    for dag in (0, 1):
        want = sum(ref.deriv(np.ascontiguousarray(A[r]), np.ascontiguousarray(B[r]), dag, mderiv=False) for r in range(nrhs))
        assert o.rel_l2(op.DhopDeriv(fa, fb, dag), want) < TOL[prec], dag
