"""FP64 refinement of a complex64 ground state at the sizes of its projections'
edges (one element, a warp, a block and the ones next to them): |dE0| <= 1e-8
(|E0| + 1), the bar of a refined energy."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,nu,nd", [((2,), 0, 0), ((2,), 1, 0), ((3,), 1, 1), ((31,), 1, 0),
                                        ((32,), 1, 0), ((11,), 1, 1), ((15,), 1, 1), ((16,), 1, 1),
                                        ((17,), 1, 1), ((6,), 3, 2), ((8,), 2, 3)])
def test_refined_energy(mb, cuda, dims, nu, nd):
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, dims), mb.PREC_F32)
    e = mb.find_min_eigenpair(op, min(150, 4 * basis.size()), reorth=True, want_vector=False,
                              refine=True).value
    exact = np.linalg.eigvalsh(oracle.hubbard_csc(list(dims), 1.0, 4.0, nu, nd).to_dense())[0]
    assert abs(e - exact) <= 1e-8 * (abs(exact) + 1)
