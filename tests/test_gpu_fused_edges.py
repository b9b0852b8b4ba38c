"""Operators whose last term rides on the hopping term's launch, and field kernels that take both
checkerboards in one launch, at odd sizes: every precision and link form (12-real and
double-float operators run the separate passes), one and several right-hand sides with padding
slots.  Bounds as in the parity tests (FP16 storage: a few roundings of 2^-11 per component)."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import MOBIUS, fermion

pytestmark = pytest.mark.gpu

TOL = {g.F64: 1e-13, g.F32: 1e-6, g.F16: 3e-3}
FORMS = [(g.F64, 0), (g.F64, g.RECON12), (g.F64, g.DF64), (g.F32, 0), (g.F32, g.RECON12), (g.F16, 0)]


def make(kind, dims, Ls, nrhs, prec, flags):
    U = g.random_gauge(dims, 0.5, 61)
    if kind == "wilson":
        return (g.WilsonFermion(U, dims, 0.1, precision=prec, nrhs=nrhs, flags=flags),
                o.OracleOp(0, 0, dims, 1, [0.1], U, g.antiperiodic_t()))
    par = [0.1, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    return (g.MobiusFermion(U, dims, Ls, *par, precision=prec, nrhs=nrhs, flags=flags),
            o.OracleOp(1, 0, dims, Ls, par, U, g.antiperiodic_t()))


@pytest.mark.parametrize("prec,flags", FORMS)
@pytest.mark.parametrize("kind,dims,Ls,nrhs", [("wilson", (2, 2, 2, 6), 1, 1), ("wilson", (4, 2, 6, 2), 1, 3),
                                               ("wilson", (4, 4, 2, 4), 1, 10), ("mobius", (2, 4, 2, 6), 6, 1),
                                               ("mobius", (4, 2, 2, 4), 14, 2)])
def test_operators_with_a_fused_term(gpu_available, kind, dims, Ls, nrhs, prec, flags):
    op, ref = make(kind, dims, Ls, nrhs, prec, flags)
    vol = int(np.prod(dims))
    names = [("M", o.OP_M), ("Mdag", o.OP_MDAG)]
    if kind == "mobius":
        names += [("Dminus", o.OP_DMINUS), ("DminusDag", o.OP_DMINUS_DAG)]
    x = fermion(vol * nrhs, Ls, 62)
    fi, fo = op.FermionField().import_(x), op.FermionField()
    for name, code in names:
        getattr(op, name)(fi, fo)
        got = fo.export().reshape(nrhs, -1)
        for r in range(nrhs):
            want = ref.apply(code, np.ascontiguousarray(x.reshape(nrhs, -1)[r]))
            assert o.rel_l2(got[r], want) < 3 * TOL[prec], (name, r)
    h = fermion(vol // 2 * nrhs, Ls, 63)
    fi, fo = op.FermionRedBlackField(g.ODD).import_(h), op.FermionRedBlackField(g.ODD)
    for name, code in (("Mpc", o.OP_MPC), ("MpcDag", o.OP_MPC_DAG)):
        getattr(op, name)(fi, fo)
        got = fo.export().reshape(nrhs, -1)
        for r in range(nrhs):
            want = ref.apply(code, np.ascontiguousarray(h.reshape(nrhs, -1)[r]), 1)
            assert o.rel_l2(got[r], want) < (10 if prec == g.F16 else 3) * TOL[prec], (name, r)


@pytest.mark.parametrize("prec", [g.F64, g.F32])
@pytest.mark.parametrize("dims,nrhs", [((2, 2, 2, 2), 1), ((2, 2, 2, 6), 3), ((4, 4, 4, 4), 7), ((6, 4, 2, 4), 16),
                                       ((8, 8, 8, 8), 1)])
def test_field_algebra_on_full_and_half_fields(gpu_available, prec, dims, nrhs):
    op, _ = make("wilson", dims, 1, nrhs, prec, 0)
    vol = int(np.prod(dims))
    for new, n in ((op.FermionField, vol), (lambda: op.FermionRedBlackField(g.ODD), vol // 2)):
        x, y = fermion(n * nrhs, 1, 64), fermion(n * nrhs, 1, 65)
        fx, fy, fz = new().import_(x), new().import_(y), new()
        x, y = fx.export().reshape(nrhs, -1), fy.export().reshape(nrhs, -1)
        tol = 1e-14 if prec == g.F64 else 1e-6
        assert np.allclose(fx.norm2(), (np.abs(x) ** 2).sum(1), rtol=tol)
        assert np.allclose(fx.inner(fy), (x.conj() * y).sum(1), rtol=tol, atol=tol * n * 12)
        g.axpby(fz, 0.5, -2.0, fx, fy)
        assert o.rel_l2(fz.export(), (0.5 * x - 2.0 * y).reshape(-1)) < tol
        n2 = g.axpy_norm(fz, 3.0, fx, fy)
        z = 3.0 * x + y
        assert o.rel_l2(fz.export(), z.reshape(-1)) < tol and np.allclose(n2, (np.abs(z) ** 2).sum(1), rtol=tol)


@pytest.mark.parametrize("prec", [g.F64, g.F32])
def test_cg_scalars_per_right_hand_side(gpu_available, prec):
    """Five right-hand sides, one of them zero (done at the start) and one with a solved guess: each
    stops on its own and the solve ends when the last one has."""
    dims, nrhs = (4, 4, 4, 6), 5
    op, ref = make("wilson", dims, 1, nrhs, prec, 0)
    vol = int(np.prod(dims))
    src = fermion(vol * nrhs, 1, 66).reshape(nrhs, -1)
    src[2] = 0
    fs, fx = op.FermionField().import_(src.reshape(-1)), op.FermionField().zero()
    tol = 1e-9 if prec == g.F64 else 1e-5
    cg = g.ConjugateGradient(tol, 2000)
    cg(g.MdagMLinearOperator(op), fs, fx)
    x = fx.export().reshape(nrhs, -1)
    assert cg.per_rhs_iterations[2] == 0 and not x[2].any()
    for r in (0, 1, 3, 4):
        assert cg.per_rhs_iterations[r] > 0
        assert o.rel_l2(ref.apply(o.OP_MDAGM, np.ascontiguousarray(x[r])), src[r]) < 3 * tol


@pytest.mark.parametrize("inner", [g.F32, g.F16])
@pytest.mark.parametrize("dims,nrhs", [((2, 2, 2, 2), 1), ((4, 2, 2, 6), 3), ((4, 4, 2, 2), 5), ((4, 4, 4, 4), 12), ((2, 2, 4, 6), 17),
                                       ((4, 2, 2, 4), 40), ((2, 2, 2, 4), 130), ((4, 4, 4, 4), 256)])
def test_wilson_schur_cg_sums_per_right_hand_side(gpu_available, inner, dims, nrhs):
    """The Schur CG whose norms and residual update ride on the hopping term: every shape of the
    per-slot sums (sites that fill a warp, that do not, one site per CTA, chunks of 16 slots)."""
    od, ref = make("wilson", dims, 1, nrhs, g.F64, 0)
    of, _ = make("wilson", dims, 1, nrhs, inner, 0)
    vol = int(np.prod(dims))
    src = fermion(vol * nrhs, 1, 67).reshape(nrhs, -1)
    fs, fx = od.FermionField().import_(src.reshape(-1)), od.FermionField()
    cg = g.ConjugateGradientReliableUpdate(1e-9, 5000, 1e-4, g.SchurDiagMooeeOperator(of), g.SchurDiagMooeeOperator(od))
    g.SchurRedBlackDiagMooeeSolve(cg)(od, fs, fx)
    x = fx.export().reshape(nrhs, -1)
    for r in sorted({0, nrhs // 2, nrhs - 1}):
        assert o.rel_l2(ref.apply(o.OP_M, np.ascontiguousarray(x[r])), src[r]) < 1e-8, r
