"""The C++ host helpers take any NTT prime below 2^62: their transforms at
primes just below 2^62, 2^61 and 2^50 equal the definition, every ring size."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "wide_modulus.cpp")
LIBDIR = os.path.join(ROOT, "gpu-resident-library_b200", "gpufhe_b200")


def test_wide_modulus(tmp_path):
    exe = str(tmp_path / "wide_modulus")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "-ccbin", "/usr/bin/g++", f"-I{ROOT}/include",
                    SRC, "-o", exe, f"-L{LIBDIR}", "-lgpufhe_b200", "-Xlinker", "-rpath", "-Xlinker", LIBDIR,
                    "-Wno-deprecated-gpu-targets"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
