"""The tiled export at its edges: fields below, at and beyond one tile of 128 5D sites, padding
right-hand sides, half and full fields, every storage precision and both canonical ones; FP32
values that the integer widening treats apart (zeros of both signs, subnormals, infinities, NaN).
An import and an export of values that the storage holds give them back bit for bit."""
import numpy as np
import pytest

import grid_gb300 as g

pytestmark = pytest.mark.gpu


def op_of(dims, Ls, nrhs, prec):
    if Ls == 1:
        return g.WilsonFermion(None, dims, 0.1, precision=prec, nrhs=nrhs)
    return g.MobiusFermion(None, dims, Ls, 0.1, 1.8, 1.5, 0.5, precision=prec, nrhs=nrhs)


@pytest.mark.parametrize("prec", [g.F64, g.F32, g.F16])
@pytest.mark.parametrize("dims,Ls,nrhs", [((2, 2, 2, 2), 1, 1), ((2, 2, 2, 4), 1, 3), ((4, 4, 2, 4), 2, 1), ((4, 2, 4, 6), 6, 2),
                                          ((4, 4, 4, 4), 1, 5), ((2, 2, 2, 10), 14, 1)])
def test_export_round_trip(gpu_available, prec, dims, Ls, nrhs):
    op = op_of(dims, Ls, nrhs, prec)
    rng = np.random.default_rng(3)
    for field in (op.FermionField(), op.FermionRedBlackField(g.ODD)):
        n = field.host_len()
        # small integers; FP16 sites get the norm 1024, which its encoder divides exactly
        x = (rng.integers(-1024, 1025, n) + 1j * rng.integers(-1024, 1025, n)).astype(np.complex128)
        x.reshape(-1, 12)[:, 0] = 1024
        field.import_(x)
        assert np.array_equal(field.export(), x)
        assert np.array_equal(field.export_f32(), x.astype(np.complex64))


def test_export_of_special_floats(gpu_available):
    op = op_of((4, 4, 4, 4), 1, 2, g.F32)
    field = op.FermionRedBlackField(g.EVEN)
    v = np.array([0.0, -0.0, 1e-45, -1e-45, 1.17549421e-38, 1.17549435e-38, -3.4028235e38, np.inf, -np.inf, np.nan, 1.0,
                  -2.5], dtype=np.float32).astype(np.float64)
    n = field.host_len()
    x = np.empty(n, dtype=np.complex128)
    x.real, x.imag = np.resize(v, n), np.resize(v[::-1], n)
    field.import_(x)
    got = field.export()
    for a, b in ((got.real, x.real), (got.imag, x.imag)):
        assert np.array_equal(a, b, equal_nan=True)
        assert np.array_equal(np.signbit(a[~np.isnan(a)]), np.signbit(b[~np.isnan(b)]))
