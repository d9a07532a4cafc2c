"""The 3 x 3 singular value decomposition behind the orthogonality Hessian
(svd3 in colb_b200/csrc/physics.cuh), from its source on the CPU: affine
matrices with off-diagonal entries of A^T A down to underflow beside equal
diagonal entries, and entries from 1e-70 to 1e70."""
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
#define HD inline
#define DV inline
using std::fabs; using std::sqrt; using std::fmax;
static double rsqrt(double x) { return 1.0 / std::sqrt(x); }
#include "vec.inc"
#include "svd.inc"
int main() {
    double A[9], U[9], s[3], V[9];
    while (std::scanf("%lf %lf %lf %lf %lf %lf %lf %lf %lf", A, A + 1, A + 2, A + 3, A + 4, A + 5, A + 6, A + 7, A + 8) == 9) {
        svd3(A, U, s, V);
        for (double v : U) std::printf("%.17g ", v);
        for (double v : s) std::printf("%.17g ", v);
        for (double v : V) std::printf("%.17g ", v);
        std::printf("\n");
    }
}
"""


def _cases():
    out = []
    for e in (0.0, 1e-16, 1e-100, 1e-160, 1e-165, 1e-170, -1e-200, 1e-300, 5e-324):
        for p in ([0, 1, 2], [1, 2, 0], [2, 0, 1], [1, 0, 2]):
            A = np.array([[1, e, 0], [0, 1, 0.1], [0, 0, 1.0]])
            out.append(A[np.ix_(p, p)])
    rng = np.random.default_rng(3)
    for scale in (1e-70, 1.0, 1e40, 1e70):
        out += [scale * rng.standard_normal((3, 3)) for _ in range(5)]
    return out


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_svd3_over_the_range_of_its_entries(tmp_path):
    d = str(tmp_path)
    src = os.path.join(ROOT, "colb_b200", "csrc")
    vec = open(os.path.join(src, "common.cuh")).read()
    open(os.path.join(d, "vec.inc"), "w").write(vec[vec.index("struct d3 {"):vec.index("HD double comp(")])
    phys = open(os.path.join(src, "physics.cuh")).read()
    open(os.path.join(d, "svd.inc"), "w").write(phys[phys.index("DV void svd3("):phys.index("// PSD projection of the Hessian of k")])
    open(os.path.join(d, "svd.cpp"), "w").write(DRIVER)
    exe = os.path.join(d, "svd")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(d, "svd.cpp"), "-o", exe])
    cases = _cases()
    text = "\n".join(" ".join("%.17g" % v for v in A.ravel()) for A in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=60, check=True).stdout
    rows = [np.array([float(v) for v in line.split()]) for line in out.splitlines()]
    assert len(rows) == len(cases)
    for A, r in zip(cases, rows):
        U, s, V = r[:9].reshape(3, 3), r[9:12], r[12:].reshape(3, 3)
        ref = np.linalg.svd(A, compute_uv=False)
        # the squares' off-diagonal part ends below 1e-17 of their trace, and a rotation's rounding is a few
        # units of 2^-53 in each of at most 16 x 3 rotations: 1e-14 of the largest value, 1e-12 where a value
        # is the root of a difference of squares (the smallest of a random matrix)
        assert np.all(np.isfinite(r)), (A, r)
        assert np.abs(np.sort(s)[::-1] - ref).max() <= 1e-12 * ref[0], (A, s, ref)
        assert np.abs((U * s) @ V.T - A).max() <= 1e-12 * ref[0], A
        assert np.abs(V.T @ V - np.eye(3)).max() <= 1e-13, A
