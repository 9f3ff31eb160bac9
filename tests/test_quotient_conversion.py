"""CPU check of the FP64-quotient basis conversion: the C++ program runs the
functions that the kernels compile in (csrc/conv_quot.hpp) for every number of sources and source width that
the library's rule admits, and compares with 128-bit arithmetic exactly."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotient_conversion(tmp_path):
    exe = tmp_path / "quotient_conversion"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "gpu-resident-library_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "quotient_conversion.cpp")], check=True)
    r = subprocess.run([str(exe), "2000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "violations=0 mismatches=0" in r.stdout
