"""The ray caster's branch-free divisions equal the IEEE division for every operand
it can pass them (all significands of the constant divisions, all arguments of
the logarithm's quotient): no tolerance."""
import ctypes
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_branch_free_divisions_are_exactly_rounded(torch_cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path / "libexact_math.so")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-std=c++17",
                        "-shared", "-Xcompiler", "-fPIC",
                        "-I", os.path.join(ROOT, "gpu-out-of-core-volume-data_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "exact_math_check.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(out)
    counts = torch_cuda.zeros(5, dtype=torch_cuda.int64, device="cuda")
    assert lib.exact_math_check(ctypes.c_void_p(counts.data_ptr()), ctypes.c_void_p(0)) == 0
    torch_cuda.cuda.synchronize()
    assert counts.tolist() == [0, 0, 0, 0, 0]
