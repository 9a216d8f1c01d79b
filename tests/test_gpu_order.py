"""Moves between the tensor and the reference order (mb_rows.h): every way an
operator's vectors cross it, against the basis's own permutation, to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one to five orbitals (high part as long as the low one, or longer), no and all
# particles of a spin, single rows and columns, tiles of one element and full
# ones with a remainder
SECTORS = [((1,), 1, 0), ((2,), 1, 1), ((3,), 2, 1), ((4,), 0, 2), ((5,), 5, 2), ((5,), 2, 3),
           ((8,), 4, 4), ((3, 3), 1, 8), ((12,), 6, 5), ((14,), 2, 7), ((4, 4), 5, 4),
           # past kTileBytes: tiles (complex128; with 6+6 every precision and both
           # sides of writes_reference)
           ((4, 4), 5, 5), ((4, 4), 9, 12), ((15,), 7, 7)]


@pytest.mark.parametrize("dims,nu,nd", SECTORS)
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_reference_order_is_the_permuted_tensor_order(mb, cuda, dims, nu, nd, prec):
    torch = cuda
    if prec == 2 and 1 in dims:
        pytest.skip("no Q64 operator with a self bond")
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 2.0, dims), prec)
    perm = torch.from_numpy(basis.permutation()).cuda()
    xt = op.seed_vector(3, order=mb.ORDER_TENSOR)
    xr = op.seed_vector(3)
    assert torch.equal(xr[perm], xt)
    assert torch.equal(op.apply(xr)[perm], op.apply(xt, order=mb.ORDER_TENSOR))
    if prec == 2:
        qt, et = op.q64_from_f64(xt, order=mb.ORDER_TENSOR)
        qr, er = op.q64_from_f64(xr)
        assert er == et and torch.equal(qr, qt)
        assert torch.equal(op.q64_to_f64(qt, et)[perm], op.q64_to_f64(qt, et, order=mb.ORDER_TENSOR))
