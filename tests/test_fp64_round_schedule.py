"""CPU check of the bound-scheduled FP64 transform rounds: the C++ program
follows csrc/fp_sched.hpp (the schedule the kernels compile in) with the
kernels' own IEEE double operations, over every round length and input bound
that occurs for 2^9 .. 2^16 points, and compares with 128-bit arithmetic. The
bounds are asserted exactly; there is no tolerance."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fp64_round_schedule(tmp_path):
    exe = tmp_path / "fp64_round_schedule"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "gpu-resident-library_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "fp64_round_schedule.cpp")], check=True)
    r = subprocess.run([str(exe), "4000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "violations=0 mismatches=0" in r.stdout
