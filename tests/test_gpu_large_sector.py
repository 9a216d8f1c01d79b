"""A sector whose vectors are far larger than L2 (1D L=16 at half filling, 166
million states): the shape a new operator starts with changes no result."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_default_shape_of_a_large_sector(mb, cuda, prec):
    torch = cuda
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(16, 16, 0)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, (16,)), prec)
    assert op.apply_shape()["prefetch"] == 1
    x = op.seed_vector(1, order=mb.ORDER_TENSOR)
    y = op.apply(x, order=mb.ORDER_TENSOR)
    op.set_apply_shape(prefetch=0)
    assert torch.equal(op.apply(x, order=mb.ORDER_TENSOR), y)
