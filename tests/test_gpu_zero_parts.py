"""complex128 applies of vectors with zero parts (real, sparse, a basis state): sums
of nothing but zeros stay on the integer pipes, and only a zero counts as one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def momentum(mb, n, k):
    basis = mb.FermionBasis.with_fixed_particle_number_spin_momentum(16, n, 0, (4, 4), k)
    return basis, mb.HubbardModelMomentum(1.0, 3.0, (4, 4))


def lattice(mb, dims, nu, nd):
    L = int(np.prod(dims))
    return (mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd),
            mb._Hubbard(1.0, 3.0, dims))


def time_us(torch, f):
    best = 1e9
    for _ in range(20):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.parametrize("kind", ["real", "imaginary", "sparse", "basis state"])
@pytest.mark.parametrize("space", ["lattice", "momentum"])
def test_zero_parts_cost_no_more(mb, cuda, space, kind):
    """Beside a full complex vector (2.5 and 1.9 times as long where zeros went to
    FP64): the look at a word of zeros is some 30 instructions beside its 150, in
    half of the words, and a sparse sum grows at any word: an eighth, and as much
    for the clock."""
    torch = cuda
    basis, model = lattice(mb, (4, 4), 4, 4) if space == "lattice" else momentum(mb, 8, (0, 0))
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F64)
    full = op.seed_vector(1)
    x = full.clone()
    if kind == "real":
        x.imag.zero_()
    elif kind == "imaginary":
        x.real.zero_()
    elif kind == "sparse":
        x[torch.rand(x.numel(), device="cuda") < 0.99] = 0
    else:
        x.zero_()
        x[x.numel() // 3] = 1
    y = op.empty()
    t = [time_us(torch, lambda v=v: op.apply(v, order=mb.ORDER_TENSOR, out=y)) for v in (full, x, full)]
    assert t[1] <= 1.25 * max(t[0], t[2]), t


@pytest.mark.parametrize("case", [((6,), 3, 3), ((3, 3), 4, 5), ((17,), 1, 8), "momentum"])
@pytest.mark.parametrize("share", [0.5, 0.9, 0.99])
def test_small_values_among_zeros(mb, cuda, case, share):
    """Zeros of both signs beside subnormals and values on both sides of 2^-511."""
    torch = cuda
    basis, model = momentum(mb, 4, (0, 1)) if case == "momentum" else lattice(mb, *case)
    m = mb.compute_matrix_elements(basis, model)
    op = mb.GpuHubbardOperator(basis, model, mb.PREC_F64)
    n = basis.size()
    rng = np.random.default_rng(n)
    x = np.zeros(n, complex)
    for part in (x.real, x.imag):
        part[:] = rng.choice([1.0, 1.25, -1.0], n)
        part *= 2.0 ** rng.choice([-1074, -1023, -1022, -700, -512, -511, -510, -40, 0], n).astype(float)
        part *= rng.random(n) >= share
    y = op.apply(torch.from_numpy(x).cuda()).cpu().numpy()
    # a row's terms and its epilogue round 2^-53 each (16 more in a momentum sector);
    # where the result is subnormal each of them 2^-1074 at most
    eps = (int(np.diff(m.row_ptr).max()) + 16) * 2.0 ** -53
    least = (int(np.diff(m.row_ptr).max()) + 16) * 2.0 ** -1074
    for got, part in ((y.real, x.real), (y.imag, x.imag)):
        t = m.values.real.astype(np.longdouble) * part[m.col_idx].astype(np.longdouble)
        full = np.flatnonzero(np.diff(m.row_ptr))
        want, size = np.zeros(n, np.longdouble), np.zeros(n, np.longdouble)
        want[full] = np.add.reduceat(t, m.row_ptr[full])
        size[full] = np.add.reduceat(np.abs(t), m.row_ptr[full])
        assert np.all(np.abs(got.astype(np.longdouble) - want) <= eps * size + least)
        assert np.all(got[size == 0] == 0)
