"""Reference-order calls captured into a CUDA graph after a first call on the stream:
nothing is left to allocate, whichever of the calls came first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one launch; the apply writes reference order (gathers, tiles); moves on both sides
@pytest.mark.parametrize("dims,nu,nd,prec", [((8,), 4, 4, 0), ((3, 4), 5, 4, 0), ((3, 4), 5, 4, 1),
                                             ((4, 4), 5, 5, 0), ((4, 4), 6, 6, 1)])
def test_affine_captured_after_an_apply(mb, cuda, dims, nu, nd, prec):
    torch = cuda
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, dims), prec)
    other = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, dims), prec)
    x, z = op.seed_vector(1), op.seed_vector(2)
    y, w = op.empty(), op.empty()
    kw = dict(scale=0.5, shift=1.5, beta=-1.0)
    want = other.apply_affine(x, z=z, **kw)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        op.apply(x, out=y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        op.apply_affine(x, z=z, out=w, **kw)
    w.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(w, want)
