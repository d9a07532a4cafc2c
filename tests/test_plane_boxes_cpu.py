"""Which bodies the line search looks at for a half-space (box_near_plane in
colb_b200/csrc/search.cu), from its source on the CPU: every body with a vertex
in the barrier's reach or a CCD bound below 1 along the step, and every body
whose swept box overflowed FP32."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
DRIVER = r"""
#include <cmath>
#include <cstdio>
#define DV inline
using std::fmin; using std::fmax;
struct float4 { float x, y, z, w; };
#include "near.inc"
int main() {
    float l[3], h[3]; double n[4], dhat, s; int ccd;
    while (std::scanf("%f %f %f %f %f %f %lf %lf %lf %lf %lf %d %lf", l, l + 1, l + 2, h, h + 1, h + 2, n, n + 1, n + 2, n + 3,
                      &dhat, &ccd, &s) == 13)
        std::printf("%d\n", (int)box_near_plane({l[0], l[1], l[2], 0}, {h[0], h[1], h[2], 0}, n, dhat, ccd, s));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_no_body_near_a_half_space_is_skipped(tmp_path):
    d = str(tmp_path)
    src = open(os.path.join(ROOT, "colb_b200", "csrc", "search.cu")).read()
    at = src.index("DV bool box_near_plane(")
    open(os.path.join(d, "near.inc"), "w").write(src[at:src.index("\n}\n", at) + 3])
    open(os.path.join(d, "near.cpp"), "w").write(DRIVER)
    exe = os.path.join(d, "near")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(d, "near.cpp"), "-o", exe])
    rng = np.random.default_rng(4)
    rows, must = [], []
    dhat, s = 0.1, 0.2
    for k in range(400):
        n = np.eye(3)[k % 3] if k % 2 else rng.standard_normal(3)
        n = n / np.linalg.norm(n)
        x = rng.uniform(-1, 1, (6, 3)) + n * rng.uniform(-1, 6)
        p = rng.uniform(-1, 1, (6, 3)) * 10.0 ** rng.uniform(-3, 1)
        if k >= 360:                                   # FP32 overflows in every direction
            p = rng.uniform(-1, 1, (6, 3)) * 1e40
            p[0], p[1] = 1e40, -1e40
        off, ccd = 0.0, k % 4 < 2
        with np.errstate(over="ignore"):
            lo = np.minimum(x, x + p).min(0).astype(np.float32) - np.float32(1e-5)
            hi = np.maximum(x, x + p).max(0).astype(np.float32) + np.float32(1e-5)
        d0, d1 = x @ n - off, (x + p) @ n - off
        near = (np.minimum(d0, d1) < dhat).any() or (ccd and (d1 < s * d0).any())
        must.append(near)
        rows.append(" ".join("%.9g" % v for v in [*lo, *hi, *n, off, dhat]) + " %d %.9g" % (ccd, s))
    out = subprocess.run([exe], input="\n".join(rows), capture_output=True, text=True, timeout=60, check=True).stdout.split()
    got = np.array([v == "1" for v in out])
    must = np.array(must)
    assert len(got) == len(must) and must[360:].all() and not must[:360].all()
    assert got[must].all()
    # an axis-parallel half-space far from a small step is skipped
    assert (~got).sum() > 40
