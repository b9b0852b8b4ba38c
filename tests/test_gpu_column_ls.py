"""The s-column programs at the even fifth dimensions between the powers and multiples of four (14,
18, 22), beside their neighbours that run the general kernels (2, 26): every 5D operator and the
Schur composites against the oracle, and the Schur CG whose residual update is a column program.
FP32 1e-6, FP16 storage 3e-3 per operator and 3e-2 for the composites, as the parity tests."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import MOBIUS, fermion

pytestmark = pytest.mark.gpu

DIMS = (2, 4, 2, 6)
TOL = {g.F32: (1e-6, 1e-6), g.F16: (3e-3, 3e-2)}


def make(Ls, prec, nrhs):
    U, par = g.random_gauge(DIMS, 0.5, 81), [0.05, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    return (g.MobiusFermion(U, DIMS, Ls, *par, precision=prec, nrhs=nrhs),
            o.OracleOp(1, 0, DIMS, Ls, par, U, g.antiperiodic_t()))


@pytest.mark.parametrize("prec", [g.F32, g.F16])
@pytest.mark.parametrize("Ls,nrhs", [(2, 1), (14, 1), (14, 3), (18, 1), (18, 2), (22, 1), (22, 5), (26, 1)])
def test_column_programs(gpu_available, prec, Ls, nrhs):
    op, ref = make(Ls, prec, nrhs)
    h = fermion(48 * nrhs, Ls, 82)
    fi, fo = op.FermionRedBlackField(g.ODD).import_(h), op.FermionRedBlackField(g.ODD)
    for k, names in enumerate(((("Mooee", o.OP_MOOEE), ("MooeeInv", o.OP_MOOEE_INV), ("MooeeInvDag", o.OP_MOOEE_INV_DAG)),
                               (("Mpc", o.OP_MPC), ("MpcDag", o.OP_MPC_DAG)))):
        for name, code in names:
            getattr(op, name)(fi, fo)
            got = fo.export().reshape(nrhs, -1)
            for r in range(nrhs):
                want = ref.apply(code, np.ascontiguousarray(h.reshape(nrhs, -1)[r]), 1)
                assert o.rel_l2(got[r], want) < TOL[prec][k], (name, r)


@pytest.mark.parametrize("prec", [g.F32, g.F16])
@pytest.mark.parametrize("Ls,nrhs", [(14, 1), (18, 2), (22, 4)])
def test_schur_cg(gpu_available, prec, Ls, nrhs):
    od, ref = make(Ls, g.F64, nrhs)
    of, _ = make(Ls, prec, nrhs)
    src = fermion(96 * nrhs, Ls, 83).reshape(nrhs, -1)
    fs, fx = od.FermionField().import_(src.reshape(-1)), od.FermionField()
    cg = g.ConjugateGradientReliableUpdate(1e-9, 20000, 1e-6, g.SchurDiagMooeeOperator(of), g.SchurDiagMooeeOperator(od),
                                           relup_every=50)
    g.SchurRedBlackDiagMooeeSolve(cg)(od, fs, fx)
    x = fx.export().reshape(nrhs, -1)
    for r in range(nrhs):
        assert o.rel_l2(ref.apply(o.OP_M, np.ascontiguousarray(x[r])), src[r]) < 1e-7, r
