"""The fixed-point form of the FP64 hopping term (grid_gb300/csrc/gb_dhop_fx.cu) on inputs whose numbers
differ in size inside one block: links, and the colours of a spinor where the links do not mix them.
FP64 arithmetic keeps each of them; the bounds are those of test_gpu_fx64.py (4e-16 over a field, 1e-15
per site)."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import fermion
from tests.test_gpu_fx64 import TOL, make
from tests.test_gpu_fx64_force_ranges import unmixed_gauge

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


@pytest.mark.parametrize("power", [1, 2, 3, 8, 32, 60])
@pytest.mark.parametrize("kind,dims,Ls,nrhs", [
    ("wilson", (4, 4, 4, 6), 1, 1), ("wilson", (6, 10, 14, 22), 1, 3), ("mobius", (4, 4, 4, 4), 6, 1),
    ("mobius", (6, 10, 10, 10), 10, 1), ("mobius", (8, 8, 6, 10), 12, 2)])
def test_colours_of_different_sizes(gpu_available, kind, dims, Ls, nrhs, power):
    """One colour 2^-power, another 2^(-2 power) of the third, on links that do not mix them: each colour of
    the result is as accurate as the largest.  Each kernel of the hopping term, and its form with the
    diagonal term (M) on a Wilson operator."""
    U = unmixed_gauge(dims, 83)
    op, ref = make(kind, dims, Ls, nrhs, U)
    vol = int(np.prod(dims))
    size = 2.0 ** -np.array([power, 0.0, 2.0 * power])
    x = (fermion(vol // 2 * nrhs, Ls, 84).reshape(-1, 3) * size).reshape(nrhs, -1)
    fi, fo = op.FermionRedBlackField(g.ODD).import_(x.reshape(-1)), op.FermionRedBlackField(g.EVEN)
    for dag in (0, 1):
        op.DhopEO(fi, fo, dag)
        got = fo.export().reshape(nrhs, -1, 3)
        for r in {0, nrhs - 1}:
            want = ref.dhop_cb(np.ascontiguousarray(x[r]), 1, dag).reshape(-1, 3)
            for c in range(3):
                assert o.rel_l2(got[r, :, c], want[:, c]) < TOL, (dag, r, c)
    if kind == "wilson":
        x = (fermion(vol * nrhs, Ls, 85).reshape(-1, 3) * size).reshape(nrhs, -1)
        fi, fo = op.FermionField().import_(x.reshape(-1)), op.FermionField()
        op.M(fi, fo)
        got = fo.export().reshape(nrhs, -1, 3)[0]
        want = ref.apply(o.OP_M, np.ascontiguousarray(x[0])).reshape(-1, 3)
        for c in range(3):
            assert o.rel_l2(got[:, c], want[:, c]) < TOL, c


@pytest.mark.parametrize("power", [32, 60])
@pytest.mark.parametrize("schur", [False, True])
@pytest.mark.parametrize("dims", [(4, 4, 4, 6), (10, 14, 18, 22)])
def test_colours_of_different_sizes_in_a_cg(gpu_available, dims, schur, power):
    """The CG's launches on one right-hand side, whose dagger reads the fixed-point copy that the launch before
    left, after three iterations against the oracle's.  Unmixed links: the iterations amplify the
    rounding of either, some 1e-15 of each colour, by less than the square of the condition number, 1e2 at
    mass 0.5 and links of modulus one."""
    U = unmixed_gauge(dims, 86)
    n = int(np.prod(dims)) // (2 if schur else 1) * 12
    x = (fermion(n // 12, 1, 87).reshape(-1, 3) * 2.0 ** -np.array([power, 0.0, power / 2])).reshape(-1)
    op = g.WilsonFermion(U, dims, 0.5)
    new = (lambda: op.FermionRedBlackField(g.ODD)) if schur else op.FermionField
    src, sol = new().import_(x), new().import_(np.zeros(n, complex))
    cg = g.ConjugateGradient(1e-30, 3, err_on_no_conv=False, check_every=1)
    cg(g.SchurDiagMooeeOperator(op) if schur else g.MdagMLinearOperator(op), src, sol)
    ref = o.OracleOp(0, 0, dims, 1, [0.5], U, g.antiperiodic_t())
    got, want = sol.export().reshape(-1, 3), ref.cg(1 if schur else 0, x, 1e-30, 3)[0].reshape(-1, 3)
    for c in range(3):
        assert o.rel_l2(got[:, c], want[:, c]) < 1e-11, c
