"""The engine's warp sums of float pairs as integers (float_fixed)."""
import os
import subprocess

from conftest import ROOT


def test_sums_are_as_exact_as_fp64_adds(tmp_path, mb):
    """Every range of terms, subnormals and the largest floats among them: exact where
    they are within 2^-32 of the largest, else within 64 units, and no further off
    than six FP64 roundings."""
    out = str(tmp_path / "float_fixed_check")
    libdir = os.path.dirname(mb.LIB_PATH)
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "float_fixed_check.cpp"),
                    "-L", libdir, "-lmanybody_gb300", f"-Wl,-rpath,{libdir}", "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
