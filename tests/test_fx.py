"""The fixed-point pair value on the host: the same functions that the kernels
compile (csrc/ds_fx.cuh), against long double.

Bound: the value is rounded once to FP64 (1.11e-16 relative at worst), and the
fixed-point steps before it stay below 2^-54 relative together: argument 3 + 2
units of 2^-56 from the squares and 4 sqrt(arg) units of 2^-61 from the
coordinates, tables 2^-56 each, polynomial and products 4 units of 2^-56; the
printed errors must stay below 1.11e-16 + 2^-53 = 2.23e-16."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fixed_point_values(tmp_path):
    exe = tmp_path / "fx_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I",
                    os.path.join(ROOT, "dachshund_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fx_check.cc"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert len(out) == 2 and all(float(v) < 2.23e-16 for v in out), out
