// physics.cuh — per-primitive device math of the ABD step.
//
//  barrier ............. barrier.py:6-65 (cubic / quadratic / log in x = d^2)
//  orthogonality ....... ortho.py:9-41
//  segment closest pts . Ericson, Real-Time Collision Detection §5.1.9, as
//                        called by contact.py:166 and abd.py:190 (float32)
//  squared distances ... IPC (Li et al. 2020) point-point, point-line,
//                        line-line and point-plane (derivatives: contact_hess.cuh)
//  triangle region ..... Ericson §5.1.5
//  additive CCD ........ Li, Kaufman, Jiang 2021 (C-IPC) Alg. 1
#pragma once
#include "common.cuh"

// ---------------------------------------------------------------- barrier
DV void barrier3(int kind, double x, double xh, double& b0, double& b1, double& b2) {
    b0 = b1 = b2 = 0.0;
    if (!(x < xh)) return;
    double t = x - xh;
    if (kind == ABD_BARRIER_CUBIC) {
        b0 = -t * t * t; b1 = -3.0 * t * t; b2 = -6.0 * t;
    } else if (kind == ABD_BARRIER_QUADRATIC) {
        b0 = t * t; b1 = 2.0 * t; b2 = 2.0;
    } else {
        double l = log(x / xh), ih = 1.0 / (xh * xh);
        b0 = -t * t * l * ih;
        b1 = (xh - x) * (2.0 * l + t / x) * ih;
        b2 = -(2.0 * l + t / x + t * (2.0 / x + xh / (x * x))) * ih;
    }
}

// ---------------------------------------------------------- orthogonality
// q: 9 doubles, rows a_i = q[3i..3i+2]
DV double ortho_energy(const double* q, double k) {
    double e = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double t = q[3*i] * q[3*j] + q[3*i+1] * q[3*j+1] + q[3*i+2] * q[3*j+2] - (i == j ? 1.0 : 0.0);
            e += t * t;
        }
    return e * k;
}
// Scale of the FP64 evaluation error of ortho_energy (in units of the
// rounding unit): k sum_ij (t_ij^2 + 4 |t_ij| |a_i| |a_j|), t_ij = a_i.a_j - delta_ij
DV double ortho_noise(const double* q, double k) {
    double na[3], e = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) na[i] = sqrt(q[3*i] * q[3*i] + q[3*i+1] * q[3*i+1] + q[3*i+2] * q[3*i+2]);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double t = q[3*i] * q[3*j] + q[3*i+1] * q[3*j+1] + q[3*i+2] * q[3*j+2] - (i == j ? 1.0 : 0.0);
            e += t * t + 4.0 * fabs(t) * na[i] * na[j];
        }
    return e * k;
}
// Scale of the FP64 evaluation error of one barrier term sc*b(x), x = d^2,
// over a stencil whose coordinates are at most L in magnitude: the term
// itself plus the barrier slope times the error of x from rounded positions
// (mult scales FP32 distances)
DV double contact_noise(double sc, double b0, double b1, double x, double L, double mult) {
    return sc * (fabs(b0) + fabs(b1) * 8.0 * sqrt(fabs(x)) * L * mult);
}
// 3x3 block (i,j) of the ortho Hessian, entry (r,c)
DV double ortho_hess(const double* q, double k, int i, int j, int r, int c) {
    double v;
    if (i == j) {
        double d = q[3*i] * q[3*i] + q[3*i+1] * q[3*i+1] + q[3*i+2] * q[3*i+2] - 1.0;
        v = q[r] * q[c] + q[3+r] * q[3+c] + q[6+r] * q[6+c] + q[3*i+r] * q[3*i+c] + (r == c ? d : 0.0);
    } else {
        double d = q[3*j] * q[3*i] + q[3*j+1] * q[3*i+1] + q[3*j+2] * q[3*i+2];
        v = q[3*j+r] * q[3*i+c] + (r == c ? d : 0.0);
    }
    return v * 4.0 * k;
}

// Singular value decomposition A = U diag(s) V^T of a 3x3 matrix (row-major):
// cyclic Jacobi on A^T A (annihilated entries set to zero), u_i = A v_i / s_i,
// a vanishing singular value's u completed by a cross product.
DV void svd3(const double* A, double* U, double* s, double* V) {
    double S[9];
#pragma unroll
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) S[3*i+j] = A[i] * A[j] + A[3+i] * A[3+j] + A[6+i] * A[6+j];
    for (int i = 0; i < 9; i++) V[i] = (i % 4 == 0) ? 1.0 : 0.0;
    const double tr = S[0] + S[4] + S[8];
    for (int sweep = 0; sweep < 16; sweep++) {
        double off = S[1] * S[1] + S[2] * S[2] + S[5] * S[5];
        if (!(off > 1e-34 * tr * tr)) break;
#pragma unroll
        for (int pq = 0; pq < 3; pq++) {
            int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            double apq = S[3*p+q];
            if (apq == 0.0) continue;
            // cot of twice the angle, then its tangent: a quotient, so that neither a tiny apq beside equal
            // diagonal entries nor large entries are squared out of range (a form without this division
            // squares both, and with |apq| below 1e-162 gives a NaN rotation)
            const double theta = (S[3*q+q] - S[3*p+p]) / (2 * apq);
            const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1));
            const double c = rsqrt(t * t + 1), sn = t * c;
            for (int k = 0; k < 3; k++) {          // S <- S R
                double skp = S[3*k+p], skq = S[3*k+q];
                S[3*k+p] = c * skp - sn * skq; S[3*k+q] = sn * skp + c * skq;
            }
            for (int k = 0; k < 3; k++) {          // S <- R^T S
                double spk = S[3*p+k], sqk = S[3*q+k];
                S[3*p+k] = c * spk - sn * sqk; S[3*q+k] = sn * spk + c * sqk;
            }
            S[3*p+q] = S[3*q+p] = 0.0;
            for (int k = 0; k < 3; k++) {          // V <- V R
                double vkp = V[3*k+p], vkq = V[3*k+q];
                V[3*k+p] = c * vkp - sn * vkq; V[3*k+q] = sn * vkp + c * vkq;
            }
        }
    }
    double smax = 0;
    for (int i = 0; i < 3; i++) { s[i] = sqrt(fmax(S[4*i], 0.0)); smax = fmax(smax, s[i]); }
    bool ok[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        ok[i] = s[i] > 1e-12 * smax && s[i] > 0.0;
        for (int r = 0; r < 3; r++)
            U[3*r+i] = ok[i] ? (A[3*r] * V[i] + A[3*r+1] * V[3+i] + A[3*r+2] * V[6+i]) / s[i] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if (ok[i]) continue;
        int j = (i + 1) % 3, k = (i + 2) % 3;
        d3 uj = mk3(U[j], U[3+j], U[6+j]), uk = mk3(U[k], U[3+k], U[6+k]);
        d3 w = cross(uj, uk);
        if (!(dot(w, w) > 0.5)) w = ok[j] ? (fabs(uj.x) < 0.9 ? cross(uj, mk3(1, 0, 0)) : cross(uj, mk3(0, 1, 0)))
                                          : mk3(i == 0, i == 1, i == 2);
        double n = sqrt(dot(w, w));
        U[i] = w.x / n; U[3+i] = w.y / n; U[6+i] = w.z / n;
        ok[i] = true;
    }
}

// PSD projection of the Hessian of k ||A A^T - I||_F^2 (A = q, entries in
// row-major order) from its analytic eigensystem: the energy is isotropic,
// psi(s) = sum (s_i^2 - 1)^2 of the singular values of A = U S V^T, and
// (Smith, de Goes, Kim 2019, "Analytic eigensystems for isotropic distortion
// energies") its nine eigenpairs are
//   U e_i e_i^T V^T                       12 s_i^2 - 4
//   U (e_i e_j^T + e_j e_i^T) V^T / sqrt2   4 (s_i^2 + s_i s_j + s_j^2 - 1)
//   U (e_i e_j^T - e_j e_i^T) V^T / sqrt2   4 (s_i^2 - s_i s_j + s_j^2 - 1)
// (times k).  usv holds U, V (row-major) and s; vec is 81 doubles of scratch.
// The lanes of a warp build the nine eigenvectors and then the entries of out
// (ld 12) times scale; all 32 call it.
struct OrthoSvd { double U[9], V[9], s[3]; };
DV void ortho_hess_psd_warp(const OrthoSvd& usv, double scale, double* vec, double* out, int lane) {
    const double r2 = 0.70710678118654752440;
    const double *U = usv.U, *V = usv.V, *s = usv.s;
    for (int e = lane; e < 81; e += 32) {
        const int m = e / 9, r = e % 9 / 3, c = e % 3;
        double v;
        if (m < 3) v = U[3*r+m] * V[3*c+m];
        else {
            const int pr = (m - 3) >> 1, i = pr == 2 ? 1 : 0, j = pr == 0 ? 1 : 2;
            const double a = U[3*r+i] * V[3*c+j], b = U[3*r+j] * V[3*c+i];
            v = ((m - 3) & 1 ? a - b : a + b) * r2;
        }
        vec[e] = v;
    }
    double lam[9];
#pragma unroll
    for (int i = 0; i < 3; i++) lam[i] = 12.0 * s[i] * s[i] - 4.0;
#pragma unroll
    for (int pr = 0; pr < 3; pr++) {
        const int i = pr == 2 ? 1 : 0, j = pr == 0 ? 1 : 2;
        lam[3 + 2 * pr] = 4.0 * (s[i] * s[i] + s[i] * s[j] + s[j] * s[j] - 1.0);
        lam[4 + 2 * pr] = 4.0 * (s[i] * s[i] - s[i] * s[j] + s[j] * s[j] - 1.0);
    }
    __syncwarp();
    for (int e = lane; e < 81; e += 32) {
        int a = e / 9, b = e % 9;
        double acc = 0;
#pragma unroll
        for (int k = 0; k < 9; k++) if (lam[k] > 0) acc += lam[k] * vec[9*k+a] * vec[9*k+b];
        out[a * 12 + b] = acc * scale;
    }
}

// ------------------------------------------------- segment closest points
// Every float operation is one IEEE round-to-nearest (no contraction), so
// the result is bit-identical to a C evaluation without FMA contraction.
DV float dotf_rn(const float* a, const float* b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a[0], b[0]), __fmul_rn(a[1], b[1])), __fmul_rn(a[2], b[2]));
}
DV float clampf01(float v) { return v < 0.f ? 0.f : (v > 1.f ? 1.f : v); }
DV void seg_seg_f32(const float* p1, const float* q1, const float* p2, const float* q2, float eps,
                    float& s, float& t, float& dist) {
    float d1[3], d2[3], r[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { d1[k] = __fsub_rn(q1[k], p1[k]); d2[k] = __fsub_rn(q2[k], p2[k]); r[k] = __fsub_rn(p1[k], p2[k]); }
    float a = dotf_rn(d1, d1), e = dotf_rn(d2, d2), f = dotf_rn(d2, r);
    if (a <= eps && e <= eps) { s = 0.f; t = 0.f; }
    else if (a <= eps) { s = 0.f; t = clampf01(__fdiv_rn(f, e)); }
    else {
        float c = dotf_rn(d1, r);
        if (e <= eps) { t = 0.f; s = clampf01(__fdiv_rn(-c, a)); }
        else {
            float b = dotf_rn(d1, d2);
            float denom = __fsub_rn(__fmul_rn(a, e), __fmul_rn(b, b));
            s = (denom != 0.f) ? clampf01(__fdiv_rn(__fsub_rn(__fmul_rn(b, f), __fmul_rn(c, e)), denom)) : 0.f;
            t = __fdiv_rn(__fadd_rn(__fmul_rn(b, s), f), e);
            if (t < 0.f) { t = 0.f; s = clampf01(__fdiv_rn(-c, a)); }
            else if (t > 1.f) { t = 1.f; s = clampf01(__fdiv_rn(__fsub_rn(b, c), a)); }
        }
    }
    float dv[3];
#pragma unroll
    for (int k = 0; k < 3; k++) dv[k] = __fsub_rn(__fadd_rn(p1[k], __fmul_rn(d1[k], s)), __fadd_rn(p2[k], __fmul_rn(d2[k], t)));
    dist = __fsqrt_rn(dotf_rn(dv, dv));
}

DV double dotd_rn(const double* a, const double* b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}
DV double clampd01(double v) { return v < 0.0 ? 0.0 : (v > 1.0 ? 1.0 : v); }
DV void seg_seg_f64(const double* p1, const double* q1, const double* p2, const double* q2, double eps,
                    double& s, double& t, double& dist) {
    double d1[3], d2[3], r[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { d1[k] = __dsub_rn(q1[k], p1[k]); d2[k] = __dsub_rn(q2[k], p2[k]); r[k] = __dsub_rn(p1[k], p2[k]); }
    double a = dotd_rn(d1, d1), e = dotd_rn(d2, d2), f = dotd_rn(d2, r);
    if (a <= eps && e <= eps) { s = 0.0; t = 0.0; }
    else if (a <= eps) { s = 0.0; t = clampd01(__ddiv_rn(f, e)); }
    else {
        double c = dotd_rn(d1, r);
        if (e <= eps) { t = 0.0; s = clampd01(__ddiv_rn(-c, a)); }
        else {
            double b = dotd_rn(d1, d2);
            double denom = __dsub_rn(__dmul_rn(a, e), __dmul_rn(b, b));
            s = (denom != 0.0) ? clampd01(__ddiv_rn(__dsub_rn(__dmul_rn(b, f), __dmul_rn(c, e)), denom)) : 0.0;
            t = __ddiv_rn(__dadd_rn(__dmul_rn(b, s), f), e);
            if (t < 0.0) { t = 0.0; s = clampd01(__ddiv_rn(-c, a)); }
            else if (t > 1.0) { t = 1.0; s = clampd01(__ddiv_rn(__dsub_rn(b, c), a)); }
        }
    }
    double dv[3];
#pragma unroll
    for (int k = 0; k < 3; k++) dv[k] = __dsub_rn(__dadd_rn(p1[k], __dmul_rn(d1[k], s)), __dadd_rn(p2[k], __dmul_rn(d2[k], t)));
    dist = __dsqrt_rn(dotd_rn(dv, dv));
}

// ------------------------------------------- point-triangle region (f64)
// 0..2 vertex, 3 edge t0t1, 4 edge t1t2, 5 edge t2t0, 6 face; IEEE ops
// without contraction, bit-identical to the C oracle.
DV int pt_region(const double* p, const double* a, const double* b, const double* c) {
    double ab[3], ac[3], ap[3], bp[3], cp[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { ab[k] = __dsub_rn(b[k], a[k]); ac[k] = __dsub_rn(c[k], a[k]); ap[k] = __dsub_rn(p[k], a[k]); }
    double d1 = dotd_rn(ab, ap), d2 = dotd_rn(ac, ap);
    if (d1 <= 0 && d2 <= 0) return 0;
#pragma unroll
    for (int k = 0; k < 3; k++) bp[k] = __dsub_rn(p[k], b[k]);
    double d3 = dotd_rn(ab, bp), d4 = dotd_rn(ac, bp);
    if (d3 >= 0 && d4 <= d3) return 1;
    double vc = __dsub_rn(__dmul_rn(d1, d4), __dmul_rn(d3, d2));
    if (vc <= 0 && d1 >= 0 && d3 <= 0) return 3;
#pragma unroll
    for (int k = 0; k < 3; k++) cp[k] = __dsub_rn(p[k], c[k]);
    double d5 = dotd_rn(ab, cp), d6 = dotd_rn(ac, cp);
    if (d6 >= 0 && d5 <= d6) return 2;
    double vb = __dsub_rn(__dmul_rn(d5, d2), __dmul_rn(d1, d6));
    if (vb <= 0 && d2 >= 0 && d6 <= 0) return 5;
    double va = __dsub_rn(__dmul_rn(d3, d6), __dmul_rn(d5, d4));
    if (va <= 0 && __dsub_rn(d4, d3) >= 0 && __dsub_rn(d5, d6) >= 0) return 4;
    return 6;
}

// ----------------------------------------------------- squared distances
// Values only (used by filters, energy and CCD).
DV double d2_pp_val(d3 a, d3 b) { d3 d = a - b; return dot(d, d); }
DV double d2_pe_val(d3 p, d3 e0, d3 e1) {
    d3 w = p - e0, e = e1 - e0; double c = dot(w, e), s = dot(e, e);
    return dot(w, w) - c * c / s;
}
DV double d2_wn_val(d3 w, d3 u, d3 v) { d3 n = cross(u, v); double a = dot(w, n); return a * a / dot(n, n); }
DV double d2_ee_line_val(d3 a0, d3 a1, d3 b0, d3 b1) { return d2_wn_val(a0 - b0, a1 - a0, b1 - b0); }
DV double d2_pt_plane_val(d3 p, d3 t0, d3 t1, d3 t2) { return d2_wn_val(p - t0, t1 - t0, t2 - t0); }

DV double pt_dist2(const double* p, const double* a, const double* b, const double* c) {
    int r = pt_region(p, a, b, c);
    d3 P = ld3(p), A = ld3(a), B = ld3(b), Cc = ld3(c);
    switch (r) {
        case 0: return d2_pp_val(P, A);
        case 1: return d2_pp_val(P, B);
        case 2: return d2_pp_val(P, Cc);
        case 3: return d2_pe_val(P, A, B);
        case 4: return d2_pe_val(P, B, Cc);
        case 5: return d2_pe_val(P, Cc, A);
        default: return d2_pt_plane_val(P, A, B, Cc);
    }
}

// ------------------------------------------------------------ additive CCD
// kind 0: edge-edge (x0 x1 | x2 x3), kind 1: point-triangle (x0 | x1 x2 x3).
// Returns 1 on a hit with *toi = conservative time; 0 if none in [0,tmax].
// The iteration count is capped at max_iter (AbdParams.ccd_max_iter, or
// ABD_CCD_MAX_ITER); on the cap the time reached so far is returned
// (conservative) and *capped is set.
DV double prim_dist2(int kind, const double* x) {
    if (kind == 0) { double s, t, d; seg_seg_f64(x, x + 3, x + 6, x + 9, 0.0, s, t, d); return d * d; }
    return pt_dist2(x, x + 3, x + 6, x + 9);
}
DV int accd(int kind, const double* x0, const double* p0, double s, double tmax, double* toi, int* capped,
            int max_iter) {
    double x[12], p[12], pm[3] = {0, 0, 0};
    for (int i = 0; i < 12; i++) { x[i] = x0[i]; p[i] = p0[i]; }
    for (int i = 0; i < 4; i++) for (int k = 0; k < 3; k++) pm[k] += p[3*i+k] * 0.25;
    for (int i = 0; i < 4; i++) for (int k = 0; k < 3; k++) p[3*i+k] -= pm[k];
    double n[4];
    for (int i = 0; i < 4; i++) n[i] = sqrt(p[3*i] * p[3*i] + p[3*i+1] * p[3*i+1] + p[3*i+2] * p[3*i+2]);
    double lp = (kind == 0) ? fmax(n[0], n[1]) + fmax(n[2], n[3]) : n[0] + fmax(n[1], fmax(n[2], n[3]));
    if (lp == 0.0) return 0;
    double d = sqrt(prim_dist2(kind, x));
    if (d == 0.0) { *toi = 0.0; return 1; }
    double g = s * d;
    double t = 0, tl = (1 - s) * d / lp;
    for (int it = 0; it < max_iter; it++) {
        for (int i = 0; i < 12; i++) x[i] += tl * p[i];
        d = sqrt(prim_dist2(kind, x));
        if (t > 0 && d < g) { *toi = t; return 1; }
        t += tl;
        if (t > tmax) return 0;
        tl = 0.9 * d / lp;
    }
    *capped = 1;
    *toi = t;
    return 1;
}
