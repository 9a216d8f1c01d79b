"""The integer hop sums' headroom (mb_isum.h): neighbours just below a power of
two, with signs that add, the first of a row a binade lower.  Floored terms then
fill a sum's 32- and 64-bit parts to the last bit."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_headroom_on_the_host(tmp_path, mb):
    """The sums restated, over the sliced tables that the apply reads."""
    out = str(tmp_path / "isum_check")
    libdir = os.path.dirname(mb.LIB_PATH)
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "isum_check.cpp"),
                    "-L", libdir, "-lmanybody_gb300", f"-Wl,-rpath,{libdir}", "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def spin_hops(dims, n):
    """(masks, target, sign) of one spin: hop k of state s goes to target[s, k] with
    sign[s, k] (0: none), every side of the lattice 3 or longer."""
    L = int(np.prod(dims))
    masks = [m for m in range(1 << L) if bin(m).count("1") == n]
    rank = {m: i for i, m in enumerate(masks)}
    stride = np.cumprod((1,) + tuple(dims))[:-1]
    bonds = []
    for i in range(L):
        for d, st in zip(dims, stride):
            x = i // st % d
            bonds.append((i, i + ((x + 1) % d - x) * st))
    rows = []
    for m in masks:
        row = []
        for a, b in bonds:
            if (m >> a & 1) == (m >> b & 1):
                continue
            lo, hi = min(a, b), max(a, b)
            between = m >> (lo + 1) & ((1 << (hi - lo - 1)) - 1)
            row.append((rank[m ^ (1 << a) ^ (1 << b)], 1 - 2 * (bin(between).count("1") & 1)))
        rows.append(row)
    width = max(map(len, rows))
    rows = [r + [(0, 0)] * (width - len(r)) for r in rows]
    t = np.array(rows, dtype=np.int64).reshape(len(masks), width, 2)
    return np.array(masks), t[:, :, 0], t[:, :, 1]


TOP, NEAR = 1 - 2.0 ** -53, 1 - 2.0 ** -40
# values of a target's down neighbours with a negative and with a positive hop
KINDS = [(-TOP, 0.4), (-NEAR, 0.4), (-TOP, TOP), (0.4, -TOP)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", range(len(KINDS)))
@pytest.mark.parametrize("dims,nu,nd", [((4, 4), 4, 4), ((4, 4), 3, 4), ((4, 4), 1, 6),
                                        ((3, 3), 4, 5), ((12,), 3, 6), ((3, 4), 6, 5)])
def test_terms_below_a_power_of_two(mb, cuda, dims, nu, nd, kind):
    torch = cuda
    L = int(np.prod(dims))
    um, ut, us = spin_hops(dims, nu)
    dm, dt, ds = spin_hops(dims, nd)
    x = np.zeros((2, len(um), len(dm)))
    # row r is made for the down state r mod D, the imaginary part with the next kind
    row, col = np.arange(len(um)), np.arange(len(um)) % len(dm)
    for part in range(2):
        neg, pos = KINDS[(kind + part) % len(KINDS)]
        for k in range(dt.shape[1]):
            v = np.select([ds[col, k] < 0, ds[col, k] > 0], [neg, pos], x[part, row, dt[col, k]])
            x[part, row, dt[col, k]] = v
    basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
    op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 3.0, dims), mb.PREC_F64)
    xd = torch.from_numpy((x[0] + 1j * x[1]).reshape(-1)).cuda()
    y = op.apply(xd, order=mb.ORDER_TENSOR).cpu().numpy().reshape(len(um), len(dm))
    both = np.array([[bin(int(a) & int(b)).count("1") for b in dm] for a in um])
    n = ut.shape[1] + dt.shape[1]
    for got, part in ((y.real, x[0]), (y.imag, x[1])):
        p = part.astype(np.longdouble)
        want = 3 * both * p
        size = np.abs(want)
        for t, s, at in ((ut, us, lambda j: p[j]), (dt, ds, lambda j: p[:, j])):
            for k in range(t.shape[1]):
                sign = s[:, k, None] if t is ut else s[None, :, k]
                term = at(t[:, k]) * sign
                want = want - term
                size = size + np.abs(term)
        # n roundings of 2^-53 of the partial sums, four in the epilogue
        assert np.all(np.abs(got - want) <= (n + 4) * 2.0 ** -53 * size)
