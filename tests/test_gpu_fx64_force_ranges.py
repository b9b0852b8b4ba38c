"""The fixed-point force term of FP64 operators (grid_gb300/csrc/gb_dhop_fx.cu) where the terms of one sum
differ in size: factors that peak at different slots, colours far below their site's largest, and
sums at the bounds of the integers.  The bounds 4e-15 per (site, direction) and 2e-15 over a field
are those of test_gpu_force_edges.py: the FP64 sums of the oracle are off by a few 1e-16 of the sum of the
terms' magnitudes, the result by no more, and the links mix at most three such sums."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import MOBIUS, fermion

pytestmark = pytest.mark.gpu


def unmixed_gauge(dims, seed):
    """Diagonal SU(3) links: the hopping term keeps the colours apart."""
    a = np.random.default_rng(seed).uniform(-np.pi, np.pi, size=(int(np.prod(dims)) * 4, 2))
    U = np.zeros((a.shape[0], 3, 3), complex)
    U[:, 0, 0], U[:, 1, 1], U[:, 2, 2] = np.exp(1j * a[:, 0]), np.exp(1j * a[:, 1]), np.exp(-1j * (a[:, 0] + a[:, 1]))
    return U.reshape(-1)


def make(dims, Ls, nrhs, U):
    if Ls == 1:
        return g.WilsonFermion(U, dims, 0.1, nrhs=nrhs), o.OracleOp(0, 0, dims, 1, [0.1], U, g.antiperiodic_t())
    par = [0.05, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    return g.MobiusFermion(U, dims, Ls, *par, nrhs=nrhs), o.OracleOp(1, 0, dims, Ls, par, U, g.antiperiodic_t())


def forces(op, ref, A, B, dag):
    """The force of A, B ([rhs][site][s][spin][colour]) and the oracle's, [site][direction][3][3]."""
    n = A.shape[0]
    fa, fb = op.FermionField().import_(A.reshape(-1)), op.FermionField().import_(B.reshape(-1))
    want = sum(ref.deriv(np.ascontiguousarray(A[r]).reshape(-1), np.ascontiguousarray(B[r]).reshape(-1), dag, mderiv=False)
               for r in range(n))
    return op.DhopDeriv(fa, fb, dag).reshape(-1, 4, 3, 3), want.reshape(-1, 4, 3, 3)


def fields(dims, Ls, nrhs, seed):
    shape = (nrhs, int(np.prod(dims)), Ls, 4, 3)
    n = int(np.prod(dims)) * nrhs
    return fermion(n, Ls, seed).reshape(shape).copy(), fermion(n, Ls, seed + 1).reshape(shape).copy()


@pytest.mark.parametrize("Ls,nrhs,d", [(12, 1, 0.3), (12, 1, 0.1), (16, 1, 0.05), (8, 1, 1e-4), (1, 3, 1e-9), (2, 9, 1e-3)])
def test_factors_that_peak_at_different_slots(gpu_available, Ls, nrhs, d):
    """A ~ d^slot and B ~ d^(slots - 1 - slot): opposite walls of the fifth dimension, or right-hand
    sides of opposite sizes.  Every slot's product is of the same size."""
    dims = (2, 4, 2, 4)
    op, ref = make(dims, Ls, nrhs, g.random_gauge(dims, 0.5, 71))
    A, B = fields(dims, Ls, nrhs, 72)
    slot = (np.arange(nrhs)[:, None] + nrhs * np.arange(Ls)[None, :])[:, None, :, None, None]
    A *= float(d) ** slot
    B *= float(d) ** (Ls * nrhs - 1 - slot)
    for dag in (0, 1):
        got, want = forces(op, ref, A, B, dag)
        err, size = np.linalg.norm(got - want, axis=(2, 3)), np.linalg.norm(want, axis=(2, 3))
        assert (err <= 4e-15 * size).all(), (dag, (err / size).max())


@pytest.mark.parametrize("power", [2, 6, 12, 40])
@pytest.mark.parametrize("Ls,nrhs", [(1, 1), (1, 2), (4, 1), (12, 1), (20, 1), (20, 2)])
def test_colours_of_different_sizes(gpu_available, Ls, nrhs, power):
    """Colours of A and B 2^-power and 2^(-2 power) of the largest, on links that do not mix them: each colour
    pair of the force is as accurate as the largest."""
    dims = (2, 4, 2, 4)
    op, ref = make(dims, Ls, nrhs, unmixed_gauge(dims, 73))
    A, B = fields(dims, Ls, nrhs, 74)
    A *= 2.0 ** -np.array([0.0, power, 2.0 * power])
    B *= 2.0 ** -np.array([power, 2.0 * power, 0.0])
    for dag in (0, 1):
        got, want = forces(op, ref, A, B, dag)
        for a in range(3):
            for b in range(3):
                assert o.rel_l2(got[:, :, a, b], want[:, :, a, b]) < 2e-15, (dag, a, b)


@pytest.mark.parametrize("Ls,nrhs", [(1, 1), (1, 2), (2, 1), (4, 1), (1, 5), (16, 1), (16, 2), (16, 4)])
def test_sums_at_the_bounds_of_the_integers(gpu_available, Ls, nrhs):
    """Every real just below a power of two, with the signs that make a projection twice that in each
    component: the largest sums that each slot count allows."""
    dims = (2, 2, 2, 4)
    op, ref = make(dims, Ls, nrhs, g.random_gauge(dims, 0.5, 75))
    x = np.zeros((nrhs, int(np.prod(dims)), Ls, 4, 3), complex)
    for signs, dag in (((1, 1, -1, 1), 0), ((1, 1, 1, -1), 1)):
        x[:] = (1 - 2.0 ** -53) * (1 + 1j) * np.array(signs)[:, None]
        got, want = forces(op, ref, x, x, dag)
        assert np.abs(got - want).max() <= 4e-15 * np.abs(want).max()
