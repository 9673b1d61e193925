"""The division of the coarse levels' updates, by a divisor whose reciprocal is at hand, is the IEEE
division bit for bit (on the host; the device's fused multiply-adds round the same way)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_divide_by_is_the_ieee_division():
    out = os.path.join(ROOT, "_build", "divide_by_test")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    cmd = [os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-O2", "--fmad=false", "-gencode",
           "arch=compute_100a,code=sm_100a", "-Xcompiler", "-ffp-contract=off", "--expt-relaxed-constexpr", "-I",
           os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "opencurrent_b200", "csrc"),
           os.path.join(ROOT, "tests", "cpp", "divide_by_test.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
