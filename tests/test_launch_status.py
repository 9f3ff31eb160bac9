"""A transform reports a refused launch of either of its two kernels: the
built object of csrc/xform.cu runs on the CPU against a stand-in for the CUDA
runtime that refuses one launch at a time."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_refused_launch_is_reported(tmp_path):
    from gpufhe_b200 import build as B
    os.makedirs(B.OBJ, exist_ok=True)
    obj = B._compile(os.path.join(B.CSRC, "xform.cu"), False)
    exe = str(tmp_path / "launch_status")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "launch_status.cpp"), obj, "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
