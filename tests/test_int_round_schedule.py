"""CPU check of the integer transform rounds that let values grow to 8q: the C++
program takes the stages that reduce from csrc/fp_sched.hpp, which the kernels
compile in, and compares with 128-bit arithmetic."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_int_round_schedule(tmp_path):
    exe = tmp_path / "int_round_bounds"
    subprocess.run(["g++", "-O2", "-std=c++17",
                    "-I" + os.path.join(ROOT, "gpu-resident-library_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "int_round_bounds.cpp")], check=True)
    r = subprocess.run([str(exe), "20000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "violations=0 mismatches=0" in r.stdout
