"""The FP64 Mpc / MpcDag whose 5D steps leave out their constant factors: every instantiated fifth
dimension and some that take the general sequence, several right-hand sides, b = 0 (whose
factor cannot be taken out), after SetMass; against the oracle at the FP64 parity bound 1e-13."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import fermion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls,nrhs,b,c", [(2, 1, 1.5, 0.5), (4, 1, 1.5, 0.5), (6, 2, 1.5, 0.5), (8, 1, 1.0, 0.0), (10, 3, 1.5, 0.5),
                                         (12, 1, 2.0, 1.0), (14, 1, 1.5, 0.5), (16, 2, 1.5, 0.5), (18, 1, 1.5, 0.5),
                                         (20, 1, 1.5, 0.5), (22, 1, 1.5, 0.5), (24, 1, 1.5, 0.5), (32, 1, 1.5, 0.5),
                                         (8, 1, 0.0, 1.0)])
def test_mpc64(gpu_available, Ls, nrhs, b, c):
    dims, U = (2, 4, 2, 6), g.random_gauge((2, 4, 2, 6), 0.5, 71)
    op = g.MobiusFermion(U, dims, Ls, 0.05, 1.8, b, c, nrhs=nrhs)
    for mass in (0.05, 0.3):
        op.SetMass(mass)
        ref = o.OracleOp(1, 0, dims, Ls, [mass, 1.8, b, c], U, g.antiperiodic_t())
        h = fermion(48 * nrhs, Ls, 72)
        fi, fo = op.FermionRedBlackField(g.ODD).import_(h), op.FermionRedBlackField(g.ODD)
        for name, code in (("Mpc", o.OP_MPC), ("MpcDag", o.OP_MPC_DAG), ("MpcDagMpc", o.OP_MPCDAGMPC)):
            getattr(op, name)(fi, fo)
            got = fo.export().reshape(nrhs, -1)
            for r in range(nrhs):
                want = ref.apply(code, np.ascontiguousarray(h.reshape(nrhs, -1)[r]), 1)
                assert o.rel_l2(got[r], want) < 1e-13, (name, mass, r)
