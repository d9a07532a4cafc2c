"""The band kernel's wide and signed instances (body bandwidths 9 to 11, and
pivots of either sign) from their source on the CPU, like
tests/test_band_kernel_cpu.py does for the narrow one."""
import os
import shutil
import subprocess

import pytest

from test_band_kernel_cpu import HERE, _kernel_source


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_wide_and_signed_band_kernels_solve_block_band_systems(tmp_path):
    d = str(tmp_path)
    open(os.path.join(d, "band_kernel.inc"), "w").write(_kernel_source())
    for f in ("simt.h", "band_wide_test.cpp"):
        shutil.copy(os.path.join(HERE, "simt", f), d)
    exe = os.path.join(d, "band_wide_test")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-pthread", os.path.join(d, "band_wide_test.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
