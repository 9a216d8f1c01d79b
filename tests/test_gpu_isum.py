"""The complex128 hop sums on the integer pipes (mb_isum.h) against sums in
extended precision, element by element: every value range they meet or hand
back to FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows of 1, 2 and 3 groups with ragged ends, a row past the staging limit
# (17 sites, 24,310 columns), 3D with doubled bonds, more than 64 hops a state
SECTORS = [((4,), 2, 1), ((6,), 3, 3), ((8,), 4, 4), ((3, 3), 4, 5), ((2, 2, 2), 4, 3),
           ((12,), 2, 6), ((17,), 1, 8), ((4, 6), 3, 2)]


def vector(kind, n, rng):
    x = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    if kind == "wide":      # 60 binades from one element to the next
        x *= 2.0 ** rng.integers(-60, 1, n)
    elif kind == "real":
        x = x.real + 0j
    elif kind == "sparse":  # most neighbourhoods hold nothing
        x[rng.random(n) < 0.99] = 0
    elif kind == "extreme":  # past what a decoded row holds, and subnormal
        x *= 2.0 ** rng.choice([-1074, -1030, -700, -512, -511, 0, 511, 512, 900], n).astype(float)
    elif kind == "growing":  # every group's largest terms come last
        x *= 2.0 ** (np.arange(n) % 97 - 48.0)
    return x


def exact(m, x):
    """(H x, sum |h||x|) of one component in extended precision, row by row."""
    t = m.values.real.astype(np.longdouble) * x[m.col_idx].astype(np.longdouble)
    full = np.flatnonzero(np.diff(m.row_ptr))
    y = np.zeros((2, m.dim), np.longdouble)
    if full.size:
        y[0, full] = np.add.reduceat(t, m.row_ptr[full])
        y[1, full] = np.add.reduceat(np.abs(t), m.row_ptr[full])
    return y


@pytest.mark.parametrize("dims,nu,nd", SECTORS)
@pytest.mark.parametrize("kind", ["uniform", "wide", "real", "sparse", "extreme", "growing"])
def test_integer_hop_sums_element_by_element(mb, cuda, dims, nu, nd, kind):
    torch = cuda
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    model = mb._Hubbard(1.0, 3.0, dims)
    m = mb.compute_matrix_elements(basis, model)
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F64)
    x = vector(kind, basis.size(), np.random.default_rng(len(kind) + nu))
    y = op.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    # n terms lose at most 2^-55 of the largest each (the integer sum), or n
    # roundings of 2^-53 of the partial sums (FP64); the epilogue rounds 4 times
    n = int(np.diff(m.row_ptr).max())
    eps = (n * 2.0 ** -53 + 4 * 2.0 ** -53)
    for got, part in ((y.real, x.real), (y.imag, x.imag)):
        want, size = exact(m, part)
        off = np.abs(got.astype(np.longdouble) - want)
        assert np.all(off <= eps * size + 4 * 2.0 ** -1074), float(np.max(off / np.maximum(size, 1e-300)))
        assert np.all(got[size == 0] == 0)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("dims,nu,nd", [((8,), 4, 4), ((3, 4), 3, 5)])
def test_non_finite_terms_reach_their_rows_only(mb, cuda, dims, nu, nd, bad):
    torch = cuda
    L = int(np.prod(dims))
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    model = mb._Hubbard(1.0, 3.0, dims)
    m = mb.compute_matrix_elements(basis, model)
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F64)
    x = vector("uniform", basis.size(), np.random.default_rng(1))
    at = basis.size() // 3
    x[at] = complex(bad, x[at].imag)
    y = op.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    values = np.zeros(m.dim)
    rows = np.repeat(np.arange(m.dim), np.diff(m.row_ptr))[m.col_idx == at]
    values[rows] = m.values.real[m.col_idx == at]
    hit = values != 0
    want = np.full(rows.size, np.nan) if np.isnan(bad) else np.sign(values[rows]) * bad
    assert np.array_equal(y.real[rows], want, equal_nan=True)
    # the rest is finite and as exact as without the value (its rows are summed
    # in FP64, so not to the last bit)
    eps = (int(np.diff(m.row_ptr).max()) + 4) * 2.0 ** -53
    x[at] = 0
    re, size = exact(m, x.real)
    assert np.all(np.abs(y.real - re)[~hit] <= eps * size[~hit])
    x[at] = complex(0, vector("uniform", basis.size(), np.random.default_rng(1))[at].imag)
    im, size = exact(m, x.imag)
    assert np.all(np.abs(y.imag - im) <= eps * size)


@pytest.mark.parametrize("kind", ["uniform", "wide", "real", "sparse", "extreme", "growing"])
@pytest.mark.parametrize("dims,n,k,lanes", [((6,), 4, (2,), 4), ((3, 3), 6, (1, 0), 4),
                                            ((4, 3), 7, (1, 2), 8), ((4, 4), 6, (0, 1), 32)])
def test_integer_row_sums_of_a_momentum_sector(mb, cuda, dims, n, k, lanes, kind):
    torch = cuda
    L, sz = int(np.prod(dims)), n % 2
    basis = mb.FermionBasis.with_fixed_particle_number_spin_momentum(L, n, sz, dims, k)
    model = mb.HubbardModelMomentum(1.0, 3.0, dims)
    m = mb.compute_matrix_elements(basis, model)
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F64)
    op.set_apply_shape(csr_lanes=lanes)
    x = vector(kind, basis.size(), np.random.default_rng(n))
    y = op.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    # as above; the lanes' sums, the off-diagonal factor and the shift round too,
    # and the diagonal is summed in another order than the exported one's
    eps = (int(np.diff(m.row_ptr).max()) + 16) * 2.0 ** -53
    for got, part in ((y.real, x.real), (y.imag, x.imag)):
        want, size = exact(m, part)
        off = np.abs(got.astype(np.longdouble) - want)
        assert np.all(off <= eps * size + 16 * 2.0 ** -1074), float(np.max(off / np.maximum(size, 1e-300)))


# (results stay normal numbers: x is 2^-20 and larger)
@pytest.mark.parametrize("k,xk", [(-975, 0), (-960, 0), (-500, -40), (300, -40), (950, 0), (950, -40)])
def test_powers_of_two_in_the_coefficients(mb, cuda, k, xk):
    """The scale of H and x powers of two: the result's exactly, also where the
    sums' own power does not fit beside the hopping's; and no hopping at all."""
    torch = cuda
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(9, 9, 1)
    one = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 8.0, (9,)), 0)
    flat = mb.GpuHubbardOperator(basis, mb._Hubbard(0.0, 8.0, (9,)), 0)
    x = one.seed_vector(2)
    want = torch.view_as_real(one.apply(x))
    got = torch.view_as_real(one.apply_affine(x * 2.0 ** xk, scale=2.0 ** k))
    assert torch.equal(got * 2.0 ** (-k // 2) * 2.0 ** (-k - -k // 2) * 2.0 ** -xk, want)
    y = flat.apply(x)
    d = (y / x).real.round()
    assert torch.equal(y, d * x) and not (d % 8).any()
