"""The check of the band solutions (band_check in colb_b200/csrc/dense.cu)
from its source on the CPU: it marks what the unpivoted factorization of an
indefinite matrix lost to a small pivot, and nothing else."""
import os
import shutil
import subprocess

import pytest

from test_band_kernel_cpu import HERE, ROOT, _kernel_source


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_solutions_that_met_a_small_pivot_are_marked(tmp_path):
    d = str(tmp_path)
    src = open(os.path.join(ROOT, "colb_b200", "csrc", "dense.cu")).read()
    open(os.path.join(d, "band_kernel.inc"), "w").write(_kernel_source())
    eng = open(os.path.join(ROOT, "colb_b200", "csrc", "engine.cuh")).read()
    find = eng[eng.index("DV int find_block("):eng.index("#define GS_LOOP")]
    open(os.path.join(d, "band_check.inc"), "w").write(find + src[src.index("constexpr double BAND_BACKWARD"):src.index("// du of every body, one warp each:")])
    for f in ("simt.h", "band_check_test.cpp"):
        shutil.copy(os.path.join(HERE, "simt", f), d)
    exe = os.path.join(d, "band_check_test")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-pthread", os.path.join(d, "band_check_test.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
