"""Applies of sectors with few rows (fewer than SMs), and of rows too long to be
staged in shared memory: their CTAs' sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(mb, dims, nu, nd, prec):
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    model = mb._Hubbard(1.0, 3.0, dims)
    return basis, model, mb.GpuHubbardOperator(basis, model, prec)


# one row to a few hundred (both sides of the SMs and of twice as many), rows of one
# column group to many, staged or not
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("dims,nu,nd", [((5,), 0, 2), ((12,), 1, 6), ((12,), 12, 5), ((14,), 2, 7), ((17,), 1, 8),
                                        ((3, 4), 2, 5), ((18,), 2, 3), ((25,), 2, 1), ((4, 4), 2, 4)])
def test_apply(mb, cuda, dims, nu, nd, prec):
    basis, model, op = operator(mb, dims, nu, nd, prec)
    H = mb.compute_matrix_elements(basis, model).to_scipy()
    x = op.seed_vector(2)
    y = op.apply(x).cpu().numpy().astype(np.complex128)
    xh = x.cpu().numpy().astype(np.complex128)
    want, size = H @ xh, abs(H) @ np.abs(xh)
    # a rounding a term of the partial sums and four in the epilogue; Q64: every
    # element to 2^-50 of the largest
    n = int(np.diff(H.indptr).max()) + 4
    off = np.maximum(np.abs((y - want).real), np.abs((y - want).imag))
    if prec == 2:
        assert np.all(off <= 2.0 ** -50 * np.abs(want).max() + n * 2.0 ** -53 * size)
    else:
        assert np.all(off <= n * 2.0 ** (-53 if prec == 0 else -24) * size)


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_few_long_rows_keep_the_gpu_busy(mb, cuda, prec):
    """17 sites 2+8 (136 rows of 24,310 columns) beside 16 sites 3+8 (560 of 12,870):
    about as long an element (three times in complex128 and Q64 with a quarter of
    the threads)."""
    torch = cuda
    per = []
    for dims, nu, nd in (((17,), 2, 8), ((16,), 3, 8)):
        _, _, op = operator(mb, dims, nu, nd, prec)
        x = op.seed_vector(1, order=mb.ORDER_TENSOR)
        if prec == 2:
            q, e = op.q64_from_f64(x, order=mb.ORDER_TENSOR)
            y = op.q64_empty()
            run = lambda: op.apply_q64(q, e, out=y)
        else:
            y = op.empty()
            run = lambda: op.apply(x, order=mb.ORDER_TENSOR, out=y)
        best = 1e9
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            run()
            a.record()
            for _ in range(5):
                run()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        per.append(best / x.numel())
    assert per[0] <= 2 * per[1], per
