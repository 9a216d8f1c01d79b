"""Lanczos recurrences that end before the steps asked for (an eigenvector, a small
invariant space): the steps queued past the end change nothing and take no time."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(mb, kind, prec):
    """An operator that is diagonal, so that every basis state is an eigenvector."""
    if kind == "momentum":
        basis = mb.FermionBasis.with_fixed_particle_number_spin_momentum(16, 8, 0, (4, 4), (1, 2))
        return mb.GpuHubbardOperator(basis, mb.HubbardModelMomentum(1.0, 0.0, (4, 4)), prec)
    if kind == "all":
        basis = mb.FermionBasis.with_fixed_particle_number(9, 8)
        return mb.GpuHubbardOperator(basis, mb._Hubbard(0.0, 3.0, (3, 3)), prec)
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(16, 8, 0)
    return mb.GpuHubbardOperator(basis, mb._Hubbard(0.0, 3.0, (4, 4)), prec)


def wall(torch, f):
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        t = time.perf_counter()
        f()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", ["lattice", "momentum", "all"])
def test_steps_past_the_end(mb, cuda, kind, prec):
    torch = cuda
    op = operator(mb, kind, prec)
    x = op.empty()
    x.zero_()
    x[x.numel() // 3] = 2
    h = op.apply(x)[x.numel() // 3].item().real / 2
    for k in (1, 2, 50, 200):
        d = mb.lanczos_pass_one(op, x, k)
        assert d.steps_taken == 1 and d.alphas.tolist() == [h] and d.b_norm == 2
    r = mb.find_min_eigenpair(op, 50, x)
    assert r.value == h
    assert torch.equal(r.vector, x)  # the Ritz vector has the start's norm
    # the next run is that of a new operator
    y = op.seed_vector(4)
    a, b = (mb.lanczos_pass_one(o, y, 4) for o in (op, operator(mb, kind, prec)))
    assert a.steps_taken == 4 and np.array_equal(a.alphas, b.alphas) and np.array_equal(a.betas, b.betas)
    if kind == "lattice":
        # two launches that return at once a step: within 15 us (an apply of this
        # sector's infinities took 130 and more)
        one, many = (wall(torch, lambda k=k: mb.lanczos_pass_one(op, x, k)) for k in (1, 60))
        assert many <= one + 59 * 15e-6, (one, many)


def test_a_run_to_the_end_of_its_space(mb, cuda):
    """Two sites, one particle of each spin: the symmetric start spans two of the four
    states (beta_1 a rounding).  More steps give the same scalars, energies, vectors."""
    torch = cuda
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(2, 2, 0)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 4.0, (2,)), mb.PREC_F64)
    x = op.empty()
    x.fill_(1.0)
    full = mb.lanczos_pass_one(op, x, 300)
    assert full.steps_taken == 2
    for k in (full.steps_taken, full.steps_taken + 1, 64, 65):
        d = mb.lanczos_pass_one(op, x, k)
        assert d.steps_taken == full.steps_taken
        assert np.array_equal(d.alphas, full.alphas) and np.array_equal(d.betas, full.betas)
    a, b = (mb.find_min_eigenpair(op, k, x) for k in (full.steps_taken, 200))
    assert a.value == b.value and torch.equal(a.vector, b.vector)
    assert torch.equal(mb.time_evolve_state(op, x, 0.3, 2), mb.time_evolve_state(op, x, 0.3, 4))
