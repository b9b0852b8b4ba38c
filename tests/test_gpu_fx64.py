"""The fixed-point form of the FP64 hopping term (grid_gb300/csrc/gb_dhop_fx.cu) at the sizes where
it can go wrong: both link layouts (below and from 8 slots per site), the split and the
one-thread-per-site kernel, remainders of warps and CTAs, padding slots; magnitudes at and
beyond the ends of its range; infinities and NaN.

Bound: the oracle sums in FP64 (measured 1.5e-16 relative L2 per site, tests/cpp/test_fx64.cpp), the
result's own rounding adds at most 2^-53, so two of them agree within 4e-16."""
import numpy as np
import pytest

import grid_gb300 as g
from oracle import oracle as o
from tests._common import MOBIUS, fermion

pytestmark = pytest.mark.gpu

TOL = 4e-16


def make(kind, dims, Ls, nrhs, U):
    if kind == "wilson":
        return (g.WilsonFermion(U, dims, 0.1, nrhs=nrhs),
                o.OracleOp(0, 0, dims, 1, [0.1], U, g.antiperiodic_t()))
    par = [0.1, MOBIUS["M5"], MOBIUS["b"], MOBIUS["c"]]
    return g.MobiusFermion(U, dims, Ls, *par, nrhs=nrhs), o.OracleOp(1, 0, dims, Ls, par, U, g.antiperiodic_t())


@pytest.mark.parametrize("kind,dims,Ls,nrhs", [
    ("wilson", (2, 2, 2, 2), 1, 1), ("wilson", (6, 2, 4, 10), 1, 1), ("wilson", (4, 4, 4, 4), 1, 7),
    ("wilson", (4, 4, 4, 6), 1, 8), ("wilson", (4, 2, 6, 4), 1, 9), ("wilson", (2, 2, 2, 4), 1, 131),
    ("mobius", (2, 4, 2, 6), 2, 1), ("mobius", (4, 4, 4, 4), 6, 1), ("mobius", (4, 6, 4, 4), 14, 1),
    ("mobius", (8, 8, 8, 8), 20, 1), ("mobius", (8, 8, 6, 10), 12, 2), ("mobius", (4, 4, 4, 4), 10, 15)])
def test_fixed_point_dhop(gpu_available, kind, dims, Ls, nrhs):
    U = g.random_gauge(dims, 0.5, 7)
    op, ref = make(kind, dims, Ls, nrhs, U)
    vol = int(np.prod(dims))
    rhs = sorted({0, nrhs // 2, nrhs - 1})
    for cb in (0, 1):
        x = fermion(vol // 2 * nrhs, Ls, 11 + cb)
        fi = op.FermionRedBlackField(cb).import_(x)
        fo = op.FermionRedBlackField(1 - cb)
        xs = x.reshape(nrhs, -1)
        for dag in (0, 1):
            (op.DhopEO if cb else op.DhopOE)(fi, fo, dag)
            y = fo.export().reshape(nrhs, -1)
            for r in rhs:
                assert o.rel_l2(y[r], ref.dhop_cb(np.ascontiguousarray(xs[r]), cb, dag)) < TOL, (cb, dag, r)
    x = fermion(vol * nrhs, Ls, 13)
    fi, fo = op.FermionField().import_(x), op.FermionField()
    for dag, code in ((0, o.OP_DHOP), (1, o.OP_DHOP_DAG)):
        op.Dhop(fi, fo, dag)
        y = fo.export().reshape(nrhs, -1)
        for r in rhs:
            assert o.rel_l2(y[r], ref.apply(code, np.ascontiguousarray(x.reshape(nrhs, -1)[r]))) < TOL, (dag, r)


@pytest.mark.parametrize("dims,Ls,nrhs", [
    ((8, 8, 6, 18), 1, 13), ((8, 8, 6, 12), 1, 19), ((8, 6, 10, 10), 12, 3), ((6, 10, 12, 10), 12, 1)])
def test_cta_sizes(gpu_available, dims, Ls, nrhs):
    """CTAs of 96 threads (12, 13 and 19 slots per site; 36 fill 128 better), 7 and 5 sites each with a remainder."""
    test_fixed_point_dhop(gpu_available, "wilson" if Ls == 1 else "mobius", dims, Ls, nrhs)


@pytest.mark.parametrize("dims,Ls,nrhs", [((10, 14, 18, 22), 1, 1), ((6, 10, 14, 22), 1, 3), ((6, 10, 10, 10), 10, 1)])
def test_two_warps_per_site(gpu_available, dims, Ls, nrhs):
    """Above 800 CTAs of 32 sites the split kernel runs two warps; the last CTA is not full."""
    test_fixed_point_dhop(gpu_available, "wilson" if Ls == 1 else "mobius", dims, Ls, nrhs)


@pytest.mark.parametrize("power", [-1060, -1000, -920, -300, 300, 870, 890, 1010])
def test_magnitudes(gpu_available, power):
    """The hopping term of 2^power x is 2^power times that of x, through the ends of the
    fixed-point range and, in FP64, beyond them (2^-1060: subnormals, absolute bound)."""
    dims, Ls = (4, 4, 4, 4), 8
    U = g.random_gauge(dims, 0.5, 8)
    op, _ = make("mobius", dims, Ls, 1, U)
    x = fermion(128, Ls, 15)
    out = []
    for scale in (1.0, 2.0 ** power if power > -1022 else 2.0 ** -1000 * 2.0 ** (power + 1000)):
        fi, fo = op.FermionRedBlackField(g.ODD).import_(x * scale), op.FermionRedBlackField(g.EVEN)
        op.DhopEO(fi, fo, 0)
        out.append(fo.export())
    back = np.ldexp(out[1].view(np.float64), -power)
    if power > -1010:
        assert o.rel_l2(back.view(np.complex128), out[0]) < TOL
    else:  # every subnormal operand and result is off by up to 2^-1075: some 200 roundings
        assert np.abs(back - out[0].view(np.float64)).max() < 200 * 2.0 ** (-1075 - power)


def test_mixed_magnitudes_zeros_and_special_values(gpu_available):
    """Sites of very different size, zero sites, one infinity and one NaN: the non-finite outputs
    are the oracle's (the neighbours of those two sites), and so is every other one."""
    dims, Ls = (4, 4, 4, 8), 4
    U = g.random_gauge(dims, 0.5, 9)
    op, ref = make("mobius", dims, Ls, 1, U)
    x = fermion(256, Ls, 17).reshape(256, Ls, 12)
    rng = np.random.default_rng(1)
    x *= 2.0 ** rng.integers(-40, 41, size=(256, 1, 1))
    x[rng.random(256) < 0.3] = 0
    clean = ref.dhop_cb(np.ascontiguousarray(x.reshape(-1)), 1, 0).reshape(256, Ls, 12)
    y = x.copy()
    y[5, 1, 3] = np.inf
    y[70, 2, 8] = np.nan
    fi, fo = op.FermionRedBlackField(g.ODD).import_(y), op.FermionRedBlackField(g.EVEN)
    op.DhopEO(fi, fo, 0)
    got = fo.export().reshape(256, Ls, 12)
    touched = ~np.isfinite(ref.dhop_cb(np.ascontiguousarray(y.reshape(-1)), 1, 0).reshape(256, Ls, 12)).all(axis=2)
    finite = np.isfinite(got).all(axis=2)
    assert (finite == ~touched).all() and touched.sum() == 16
    scale = np.linalg.norm(clean, axis=2)
    err = np.linalg.norm(np.where(finite[..., None], got - clean, 0), axis=2)
    assert (err <= 1e-15 * scale).all()  # per site; sites without neighbours are exactly zero


def test_links_of_any_size_and_reimport(gpu_available):
    """Gauge fields that are not unitary: the links' exponent follows them, and an import replaces
    the copies; links of zeros and beyond the range use the FP64 kernel."""
    dims, Ls = (4, 4, 4, 4), 8
    U = g.random_gauge(dims, 0.5, 10)
    op, _ = make("mobius", dims, Ls, 1, U)
    x = fermion(128, Ls, 19)
    fi, fo = op.FermionRedBlackField(g.ODD).import_(x), op.FermionRedBlackField(g.EVEN)
    op.DhopEO(fi, fo, 0)
    one = fo.export()
    for scale in (3.0, 1e-3, 1e12, 0.0, 1.0):
        op.ImportGauge(U * scale)
        op.DhopEO(fi, fo, 0)
        assert np.abs(fo.export() - scale * one).max() <= 4e-15 * scale * np.abs(one).max()


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 4, 4, 6), (6, 2, 4, 10), (8, 8, 8, 8), (10, 14, 18, 22)])
@pytest.mark.parametrize("tiny", [False, True])
@pytest.mark.parametrize("schur", [False, True])
def test_cg_sums_in_the_hopping_term(gpu_available, dims, tiny, schur):
    """One right-hand side takes the CG's sums and residual update in the hopping term's launch, two
    the separate passes: the same solution and iterations.  tiny: a point source and values
    below the fixed-point range elsewhere, so that both kinds of site end in a sum.  Bound: both
    true residuals are below 1e-10, the condition number of M^dag M (mass 0.5) below 1000."""
    U = g.random_gauge(dims, 0.5, 17)
    n = int(np.prod(dims)) // (2 if schur else 1) * 12
    x = fermion(n // 12, 1, 18)
    if tiny:
        x = x.copy()
        x[12:] *= 2.0 ** -940
    got = []
    for nrhs in (1, 2):
        op = g.WilsonFermion(U, dims, 0.5, nrhs=nrhs)
        new = (lambda: op.FermionRedBlackField(g.ODD)) if schur else op.FermionField
        src, sol = new().import_(np.concatenate([x] * nrhs)), new().import_(np.zeros(n * nrhs, complex))
        cg = g.ConjugateGradient(1e-10, 500, check_every=1)
        cg(g.SchurDiagMooeeOperator(op) if schur else g.MdagMLinearOperator(op), src, sol)
        got.append((sol.export().reshape(nrhs, -1)[0], cg.IterationsToComplete))
    assert abs(got[0][1] - got[1][1]) <= 1
    assert o.rel_l2(got[0][0], got[1][0]) < 2e-7
