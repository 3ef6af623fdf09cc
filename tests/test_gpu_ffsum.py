"""The sums and scalars of the persistent structured solve are FP64 from the warps up,
the batched step's as good as FP64 (csrc/ds_ffsum.cuh): tests/cpp/ffsum_check.cu runs
its functions on the device and prints each error beside the bound derived there."""
import os
import subprocess

import pytest

from dachshund_gb300.build import ARCH, CSRC, INCLUDE, nvcc

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_sums_and_scalars(tmp_path):
    exe = str(tmp_path / "ffsum_check")
    subprocess.run([nvcc()] + ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr",
                                      "-I" + INCLUDE, "-I" + CSRC, "-o", exe,
                                      os.path.join(HERE, "cpp", "ffsum_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    lines = [ln.split() for ln in out.splitlines()]
    assert len(lines) == 10, out
    for name, err, bound in lines:
        assert float(err) <= float(bound), out
