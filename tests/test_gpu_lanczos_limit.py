"""Lanczos runs whose step limit is a bound that they do not reach, and runs longer
than the device scalars' first room (1,024 steps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(mb, prec, dims=(8,), nu=4, nd=4):
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(int(np.prod(dims)), nu + nd, nu - nd)
    return mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, dims), prec)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("k", [10 ** 6, 10 ** 12, 2 ** 62])
def test_a_limit_that_is_not_reached(mb, cuda, prec, k):
    op = operator(mb, prec)
    kw = dict(conv_tol=1e-9, check_every=10, want_vector=True)
    a = mb.find_min_eigenpair(op, 300, op.seed_vector(1), **kw)
    b = mb.find_min_eigenpair(op, k, op.seed_vector(1), **kw)
    assert a.steps == b.steps < 300 and a.value == b.value
    assert cuda.equal(a.vector, b.vector)


@pytest.mark.parametrize("every", [1, 63, 64, 65, 100, 2 ** 31 - 1])
def test_checks_between_the_looks(mb, cuda, every):
    """A run stops at a multiple of check_every, wherever the scalars are looked at."""
    op = operator(mb, 0)
    r = mb.find_min_eigenpair(op, 260, op.seed_vector(1), conv_tol=1e-10, check_every=every,
                              want_vector=False)
    assert r.steps % every == 0 or r.steps == 260


@pytest.mark.parametrize("k", [1023, 1024, 1025, 2100])
def test_long_runs(mb, cuda, k):
    """complex64 goes on past every eigenvalue: the same scalars whatever the limit,
    and a replay of all of them."""
    op = operator(mb, 1)
    x = op.seed_vector(3)
    d, e = mb.lanczos_pass_one(op, x, k), mb.lanczos_pass_one(op, x, 2200)
    assert d.steps_taken == k
    assert np.array_equal(d.alphas, e.alphas[:k]) and np.array_equal(d.betas, e.betas[:k - 1])
    y = np.zeros(k, complex)
    y[0] = d.b_norm
    assert cuda.allclose(mb.lanczos_pass_two(op, x, d, y), x, rtol=1e-6, atol=0)
