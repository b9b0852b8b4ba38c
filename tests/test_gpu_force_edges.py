"""The force kernels at their edges: sites that do not fill a warp, a single vector along s (one lane
per site), uneven walks of the two lanes, several right-hand sides with a padding slot; for the
FP64 operators' fixed-point form each width of its limbs, the slot count above which the FP64
kernel runs, magnitudes at and beyond its range, infinities and NaN.  FP64 relative L2 1e-13, FP32
1e-6, as the operators' parity bounds; where a bound of 2e-15 stands, the oracle's FP64 sums of up
to 64 x 24 terms are off by a few 1e-16 and the result by less."""
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


@pytest.mark.parametrize("Ls,nrhs", [(16, 1), (2, 9), (16, 2), (10, 4), (16, 4), (22, 3)])
def test_force_fp64_slot_counts(gpu_available, Ls, nrhs):
    dims, U, ph = (2, 2, 4, 2), g.random_gauge((2, 2, 4, 2), 0.5, 54), g.antiperiodic_t()
    par = [0.05, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    op, ref = g.MobiusFermion(U, dims, Ls, *par, nrhs=nrhs), o.OracleOp(1, 0, dims, Ls, par, U, ph)
    A, B = fermion(32 * nrhs, Ls, 55).reshape(nrhs, -1), fermion(32 * nrhs, Ls, 56).reshape(nrhs, -1)
    fa, fb = op.FermionField().import_(A.reshape(-1)), op.FermionField().import_(B.reshape(-1))
    for dag in (0, 1):
        want = sum(ref.deriv(np.ascontiguousarray(A[r]), np.ascontiguousarray(B[r]), dag, mderiv=False) for r in range(nrhs))
        assert o.rel_l2(op.DhopDeriv(fa, fb, dag), want) < 2e-15, dag


@pytest.mark.parametrize("pa,pb", [(-900, 0), (0, 870), (900, -900), (-930, 0), (-440, -440), (-455, -455), (445, 445),
                                   (460, 460)])
def test_force_fp64_magnitudes(gpu_available, pa, pb):
    dims, Ls = (2, 2, 4, 2), 6
    op = g.MobiusFermion(g.random_gauge(dims, 0.5, 57), dims, Ls, 0.05, 1.8, 1.5, 0.5)
    A, B = fermion(32, Ls, 58), fermion(32, Ls, 59)
    out = []
    for a, b in ((A, B), (A * 2.0 ** pa, B * 2.0 ** pb)):
        fa, fb = op.FermionField().import_(a), op.FermionField().import_(b)
        out.append(op.DhopDeriv(fa, fb, 0))
    assert o.rel_l2(np.ldexp(out[1].view(np.float64), -pa - pb).view(np.complex128), out[0]) < 2e-15


def test_force_fp64_zeros_and_special_values(gpu_available):
    dims, Ls, vol = (2, 2, 4, 4), 4, 64
    U, ph = g.random_gauge(dims, 0.5, 60), g.antiperiodic_t()
    par = [0.05, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    op, ref = g.MobiusFermion(U, dims, Ls, *par), o.OracleOp(1, 0, dims, Ls, par, U, ph)
    rng = np.random.default_rng(2)
    A, B = fermion(vol, Ls, 61).reshape(vol, Ls, 12), fermion(vol, Ls, 62).reshape(vol, Ls, 12)
    A *= 2.0 ** rng.integers(-30, 31, size=(vol, 1, 1))
    A[rng.random(vol) < 0.3] = 0
    A[7, 2, 5], B[40, 1, 3] = np.inf, np.nan
    fa, fb = op.FermionField().import_(A.reshape(-1)), op.FermionField().import_(B.reshape(-1))
    got = op.DhopDeriv(fa, fb, 0).reshape(vol, 4, 9)
    want = ref.deriv(A.reshape(-1).copy(), B.reshape(-1).copy(), 0, mderiv=False).reshape(vol, 4, 9)
    ok, fin = np.isfinite(want).all(axis=2), np.isfinite(got).all(axis=2)
    assert (ok == fin).all() and 5 <= (~ok).sum() <= 8
    err = np.linalg.norm(np.where(ok[..., None], got - want, 0), axis=2)
    assert (err <= 4e-15 * np.linalg.norm(np.where(ok[..., None], want, 0), axis=2)).all()
