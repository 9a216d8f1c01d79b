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


# both sides of one_launch, odd rows, rows too long for shared memory, one row
@pytest.mark.parametrize("prec,dims,nu,nd", [
    (0, (2,), 1, 1), (0, (3, 3), 4, 5), (0, (5,), 5, 2), (0, (1,), 1, 0), (0, (20,), 0, 10),
    (0, (18,), 2, 3), (0, (4, 4), 3, 3), (1, (3, 3), 4, 5), (1, (20,), 10, 0), (1, (18,), 1, 9),
    (1, (20,), 0, 9), (1, (20,), 0, 10)])
def test_one_launch_calls_are_the_permuted_tensor_order(mb, cuda, prec, dims, nu, nd):
    torch = cuda
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 2.0, dims), prec)
    perm = torch.from_numpy(basis.permutation()).cuda()
    x, z = op.seed_vector(3), op.seed_vector(4)
    if x.numel() > 1:
        x[x.numel() // 2] = float("inf")
    want = op.apply_affine(x[perm], scale=0.5, shift=0.25, beta=-2.0, z=z[perm],
                           order=mb.ORDER_TENSOR)

    def same(got):
        return torch.equal(torch.view_as_real(got[perm]).isnan(), torch.view_as_real(want).isnan()) \
            and torch.equal(torch.view_as_real(got[perm]).nan_to_num(7.0),
                            torch.view_as_real(want).nan_to_num(7.0))

    assert same(op.apply_affine(x, scale=0.5, shift=0.25, beta=-2.0, z=z))
    y = z.clone()
    assert same(op.apply_affine(x, scale=0.5, shift=0.25, beta=-2.0, z=y, out=y))
    # x and y, z and y in one buffer, one element apart
    n = x.numel()
    buf = torch.empty(n + 1, dtype=x.dtype, device=x.device)
    buf[1:] = x
    assert same(op.apply_affine(buf[1:], scale=0.5, shift=0.25, beta=-2.0, z=z, out=buf[:n]))
    buf[1:] = z
    assert same(op.apply_affine(x, scale=0.5, shift=0.25, beta=-2.0, z=buf[1:], out=buf[:n]))
