"""The complex64 apply's rows: up lists read four entries at a time and sliced
tables ordered for 8-byte elements, against an FP64 sum, where they can go
wrong: odd row lengths (the list's alignment after the row), lists of every
remainder modulo four with the signs changing anywhere, one to three column
groups, rows too long to stage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [((5,), 2, 2), ((7,), 3, 1), ((3, 3), 4, 3), ((9,), 4, 4), ((2, 5), 3, 4), ((11,), 5, 2),
           ((3, 4), 5, 4), ((2, 2, 3), 6, 5), ((13,), 3, 6), ((17,), 1, 8)]


@pytest.mark.parametrize("dims,nu,nd", SECTORS)
def test_complex64_rows(mb, cuda, dims, nu, nd):
    torch = cuda
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    model = mb._Hubbard(1.0, 3.0, dims)
    H = mb.compute_matrix_elements(basis, model).to_scipy()
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F32)
    x = op.seed_vector(5)
    y = op.apply(x).cpu().numpy().astype(np.complex128)
    xh = x.cpu().numpy().astype(np.complex128)
    want = H @ xh
    size = abs(H) @ np.abs(xh)
    # one rounding of 2^-24 of the partial sums a term, four in the epilogue
    eps = (int(np.diff(H.indptr).max()) + 4) * 2.0 ** -24
    for got, ref in ((y.real, want.real), (y.imag, want.imag)):
        assert np.all(np.abs(got - ref) <= eps * size)
