"""Moves between the tensor and the reference order of lopsided sectors, whose tiles
would hold few elements (order_tile_count, kTileFill)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_tile_count(tmp_path, mb):
    out = str(tmp_path / "order_check")
    libdir = os.path.dirname(mb.LIB_PATH)
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "order_check.cpp"),
                    "-L", libdir, "-lmanybody_gb300", f"-Wl,-rpath,{libdir}", "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def best_us(torch, f):
    best = 1e9
    for _ in range(6):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        f()
        a.record()
        f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.gpu
def test_lopsided_moves(mb, cuda):
    """22 sites 11+1 (39 elements a tile) beside 4x4 5+5: within three times as long an
    element (six by tiles), and the permuted tensor order to the bit."""
    torch = cuda
    per = []
    for dims, nu, nd in (((22,), 11, 1), ((4, 4), 5, 5)):
        L = int(np.prod(dims))
        basis = mb.FermionBasis.with_fixed_particle_number_and_spin(L, nu + nd, nu - nd)
        op = mb.GpuHubbardOperator(basis, mb._Hubbard(1.0, 2.0, dims), mb.PREC_Q64)
        xr = op.seed_vector(3)
        q, e = op.q64_from_f64(xr)
        if nu == 11:
            perm = torch.from_numpy(basis.permutation()).cuda()
            qt, et = op.q64_from_f64(xr[perm], order=mb.ORDER_TENSOR)
            assert et == e and torch.equal(q, qt)
            assert torch.equal(op.q64_to_f64(q, e)[perm], op.q64_to_f64(q, e, order=mb.ORDER_TENSOR))
            del perm, qt
        y = op.empty()
        per.append(best_us(torch, lambda: (op.q64_from_f64(xr, out=q), op.q64_to_f64(q, e, out=y))) / xr.numel())
    assert per[0] <= 3 * per[1], per
