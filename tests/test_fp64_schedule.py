"""CPU check of the FP64 NTT butterfly schedule for unsigned twiddles (the
reference's tables: normalisations after every second stage): exact against
128-bit modular arithmetic, with every magnitude stated in csrc/ntt.cuh
asserted, on random and adversarial inputs. The C++ program takes the schedule
from csrc/fp_sched.hpp and performs the kernel's own IEEE double operations, so
a pass here means the device path computes the same residues."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fp64_butterfly_schedule(tmp_path):
    exe = tmp_path / "fp64_unsigned_rounds"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "gpu-resident-library_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "fp64_unsigned_rounds.cpp")], check=True)
    r = subprocess.run([str(exe), "60000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "violations=0 mismatches=0" in r.stdout
