"""The contacts' Hessians in five directions and their 5 x 5 projection
(stencil_hessian, psd_project5 and contact_matrix5 in
colb_b200/csrc/contact_hess.cuh), from their source on the CPU, against the
second derivatives of the squared distances by automatic differentiation and an
eigen-decomposition of the whole matrix: every stencil type, both modes,
repeated and vanishing eigenvalues, touching points and a half-space without a
normal."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PP, PE, EE, PT, PG = range(5)
NP = {PP: 2, PE: 3, EE: 4, PT: 4, PG: 1}
DRIVER = r"""
#include <cmath>
#include <cstdio>
#define DV inline
#define HD inline
#define T_PP 0
#define T_PE 1
#define T_EE 2
#define T_PT 3
#define T_PG 4
using std::fabs; using std::sqrt; using std::fmax; using std::fma;
static double rsqrt(double x) { return 1.0 / std::sqrt(x); }
#include "hess.inc"
int main() {
    int type, projected;
    double v[12], pl[4], B1, B2;
    while (std::scanf("%d %d", &type, &projected) == 2) {
        for (double& a : v) if (std::scanf("%lf", &a) != 1) return 1;
        for (double& a : pl) if (std::scanf("%lf", &a) != 1) return 1;
        if (std::scanf("%lf %lf", &B1, &B2) != 2) return 1;
        d3 x[4];
        for (int i = 0; i < 4; i++) x[i] = mk3(v[3*i], v[3*i+1], v[3*i+2]);
        Stencil5 S;
        stencil_hessian(type, x, pl, S);
        contact_matrix5(type, projected, B1, B2, S);
        const double *w[5] = {S.c, S.b2, S.b3, S.c, S.c}, *dir[5] = {S.n, S.n, S.n, S.e1, S.e2};
        double u[5][12];
        for (int p = 0; p < 5; p++) for (int i = 0; i < 12; i++) u[p][i] = w[p][i / 3] * dir[p][i % 3];
        for (int i = 0; i < 12; i++) std::printf("%.17g ", 2.0 * S.d * S.cn * B1 * u[0][i]);
        for (int i = 0; i < 12; i++)
            for (int j = 0; j < 12; j++) {
                double h = 0;
                for (int p = 0; p < 5; p++) for (int q = 0; q < 5; q++) h += S.a[s5(p, q)] * u[p][i] * u[q][j];
                std::printf("%.17g ", h);
            }
        std::printf("\n");
    }
}
"""


def _square(torch, type_, x, pl):
    def wn(w, u, v):
        n = torch.linalg.cross(u, v)
        return (w @ n) ** 2 / (n @ n)
    if type_ == PG:
        return (pl[:3] @ x[0] - pl[3]) ** 2
    if type_ == PP:
        return (x[0] - x[1]) @ (x[0] - x[1])
    if type_ == PE:
        w, e = x[0] - x[1], x[2] - x[1]
        return w @ w - (w @ e) ** 2 / (e @ e)
    if type_ == EE:
        return wn(x[0] - x[2], x[1] - x[0], x[3] - x[2])
    return wn(x[0] - x[1], x[2] - x[1], x[3] - x[1])


def _psd(H):
    w, V = np.linalg.eigh((H + H.T) / 2)
    return (V * np.maximum(w, 0)) @ V.T


def _cases():
    rng = np.random.default_rng(12)
    out = []

    def add(type_, x, pl, B1, B2):
        for projected in (0, 1):
            out.append((type_, projected, np.asarray(x, float), np.asarray(pl, float), B1, B2))
    up = [0.0, 1.0, 0.0, -0.4]
    for type_ in (PP, PE, EE, PT, PG):
        for k in range(25):
            n = rng.standard_normal(3)
            B1, B2 = -10.0 ** rng.uniform(-3, 6), 10.0 ** rng.uniform(-3, 12)
            if k % 5 == 4:
                B1 = -B1                       # (a quadratic barrier's slope has one sign, the projection may not need it)
            add(type_, rng.standard_normal((4, 3)), [*(n / np.linalg.norm(n)), rng.normal()], B1, B2)
    # symmetric stencils: repeated eigenvalues; slopes that put one at zero
    cross = [[-1, 0, 0.3], [1, 0, 0.3], [0, -1, 0], [0, 1, 0]]
    tri = [[0, 0.2, 0], [-1, 0, -1], [1, 0, -1], [0, 0, 1]]
    for B1, B2 in ((-1.0, 0.0), (-1.0, 2.0), (1.0, -1.0), (0.0, 1.0), (-2.0, 1.0 / 0.09), (0.0, 0.0)):
        add(EE, cross, up, B1, B2)
        add(PT, tri, up, B1, B2)
        add(PE, [[0, 0.1, 0], [-1, 0, 0], [1, 0, 0], [0, 0, 0]], up, B1, B2)
        add(PP, [[0, 0.1, 0], [0, 0, 0], [0, 0, 0], [0, 0, 0]], up, B1, B2)
        add(PG, [[0.2, 0.3, -0.1], [0, 0, 0], [0, 0, 0], [0, 0, 0]], up, B1, B2)
    add(PP, [[1e-9, 0, 0], [0, 0, 0], [0, 0, 0], [0, 0, 0]], up, -1.0, 1e6)
    add(PG, [[0.2, 0.3, -0.1], [0, 0, 0], [0, 0, 0], [0, 0, 0]], [0, 0, 0, 0.5], -1.0, 2.0)     # no normal
    add(PG, [[0.2, 0.3, -0.1], [0, 0, 0], [0, 0, 0], [0, 0, 0]], [0, 2.5, 0, 0.1], -1.0, 2.0)   # not of length 1
    return out


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_contact_hessians_and_their_projection(tmp_path):
    import torch
    d = str(tmp_path)
    src = lambda f: open(os.path.join(ROOT, "colb_b200", "csrc", f)).read()
    common = src("common.cuh")
    text = common[common.index("struct d3 {"):common.index("HD double comp(")]
    text += src("contact_hess.cuh").replace("#pragma once", "").replace('#include "common.cuh"', "")
    open(os.path.join(d, "hess.inc"), "w").write(text)
    open(os.path.join(d, "hess.cpp"), "w").write(DRIVER)
    exe = os.path.join(d, "hess")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(d, "hess.cpp"), "-o", exe])
    cases = _cases()
    lines = ["%d %d " % c[:2] + " ".join("%.17g" % v for v in [*c[2].ravel(), *c[3], c[4], c[5]]) for c in cases]
    out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, timeout=120, check=True).stdout
    rows = [np.array([float(v) for v in line.split()]) for line in out.splitlines()]
    assert len(rows) == len(cases)
    for (type_, projected, x, pl, B1, B2), r in zip(cases, rows):
        n = 3 * NP[type_]
        xt, plt = torch.tensor(x.ravel()[:n]), torch.tensor(pl)
        f = lambda y: _square(torch, type_, y.reshape(-1, 3), plt)
        g = torch.autograd.functional.jacobian(f, xt).numpy()
        F = torch.autograd.functional.hessian(f, xt).numpy()
        gg = B2 * np.outer(g, g)
        if projected:
            H = _psd(B1 * F + gg)
        else:
            H = (0 if type_ == PP else B1) * (_psd(F) if type_ == EE else F) + gg
        got_g, got = r[:12][:n], r[12:].reshape(12, 12)[:n, :n]
        assert np.all(np.isfinite(r)), (type_, projected, x, pl)
        # both sides round their terms, |B1| |f''| + |B2| |g|^2 at most, in a few hundred operations; the random
        # stencils' edges come within about 3 degrees of parallel, which multiplies that by up to 1 / sin^2 = 400
        scale = abs(B1) * np.abs(F).max() + abs(B2) * (g @ g)
        assert np.abs(got - H).max() <= 1e-10 * scale, (type_, projected, x, B1, B2)
        assert np.abs(got_g - B1 * g).max() <= 1e-10 * abs(B1) * max(np.abs(g).max(), 1e-300), (type_, x)
        assert np.abs(r[12:].reshape(12, 12)[n:]).max(initial=0) == 0
