// contact_hess.cuh — the barrier Hessian of one contact in closed form up to a
// 5 x 5 eigenproblem.
//
// A squared distance f = d^2 of a stencil (point-point, point-edge, line-line,
// point-plane) changes to second order only through
//   s = sum_i c_i dx_i      the relative displacement of the closest points
//                           (c: the closest points' weights, summing to zero),
//   p                       the rotation of the normal n, linear in the
//                           normal parts of the edges' displacements:
//   f = d^2 + 2 d s.n + (s.n)^2 + 2 d s.p - d^2 |p|^2 + O(3)
// (for point-edge the rotation is that of the edge, and the part of s across
// the edge and n adds its square).  So its Hessian lives on the five
// orthonormal directions
//   c (x) n, b2 (x) n, b3 (x) n, c (x) e1, c (x) e2
// (c normalised; b2, b3 complete the edges' weights; e1, e2 span the plane
// normal to n), the gradient is 2 d |c| along the first, and projecting the
// 12 x 12 barrier Hessian onto the PSD cone is projecting a 5 x 5 matrix.
// A 12 x 12 cyclic Jacobi over a warp took 66 to 88 rounds of 2,200 cycles per
// contact; the 5 x 5 one runs in registers without shuffles.
#pragma once
#include "common.cuh"

struct Stencil5 {
    double n[3], e1[3], e2[3];   // frame
    double c[4], b2[4], b3[4];   // weights per vertex, orthonormal
    double d, cn;                // distance, |c| before normalisation
    double a[15];                // Hessian of f in the five directions, upper triangle by rows
};
HD constexpr int s5(int i, int j) { return i <= j ? i * 5 - i * (i - 1) / 2 + (j - i) : s5(j, i); }

DV double dot4(const double* a, const double* b) { return a[0]*b[0] + a[1]*b[1] + a[2]*b[2] + a[3]*b[3]; }
// v minus its parts along the unit vectors a (and b), normalised
DV void orth4(const double* v, const double* a, const double* b, double* o) {
    const double ta = dot4(v, a), tb = b ? dot4(v, b) : 0.0;
    double s = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) { o[i] = v[i] - ta * a[i] - (b ? tb * b[i] : 0.0); s += o[i] * o[i]; }
    const double is = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] *= is;
}
DV void store3(double* o, d3 v) { o[0] = v.x; o[1] = v.y; o[2] = v.z; }
// unit vectors e1, e2 with (e1, e2, n) orthonormal
DV void perp_frame(d3 n, d3& e1, d3& e2) {
    const double ax = fabs(n.x), ay = fabs(n.y), az = fabs(n.z);
    const d3 k = ax <= ay && ax <= az ? mk3(1, 0, 0) : (ay <= az ? mk3(0, 1, 0) : mk3(0, 0, 1));
    e1 = cross(n, k);
    e1 = (1.0 / sqrt(dot(e1, e1))) * e1;
    e2 = cross(n, e1);
}

// type T_*; x: the stencil's vertices (for T_PG the vertex, with the plane's
// normal and offset in pl)
DV void stencil_hessian(int type, const d3* x, const double* pl, Stencil5& S) {
#pragma unroll
    for (int i = 0; i < 15; i++) S.a[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) { S.c[i] = 0.0; S.b2[i] = 0.0; S.b3[i] = 0.0; }
    d3 n, e1, e2;
    if (type == T_PG) {
        n = mk3(pl[0], pl[1], pl[2]);
        S.d = dot(n, x[0]) - pl[3];
        S.c[0] = 1.0; S.cn = 1.0;
        e1 = e2 = mk3(0, 0, 0);                     // nothing but n; a frame would divide by its length, which may be 0
        S.a[s5(0, 0)] = 2.0;
    } else if (type == T_PP) {
        const d3 r = x[0] - x[1];
        S.d = sqrt(dot(r, r));
        n = S.d > 0.0 ? (1.0 / S.d) * r : mk3(1, 0, 0);
        perp_frame(n, e1, e2);
        const double h = 0.70710678118654752440;
        S.cn = 1.41421356237309504880; S.c[0] = h; S.c[1] = -h;
        S.a[s5(0, 0)] = S.a[s5(3, 3)] = S.a[s5(4, 4)] = 4.0;
    } else if (type == T_PE) {
        const d3 w = x[0] - x[1], e = x[2] - x[1];
        const double ee = dot(e, e), il = 1.0 / sqrt(ee), g = dot(w, e) / ee;
        e1 = il * e;
        const d3 r = w - g * e;
        S.d = sqrt(dot(r, r));
        if (S.d > 0.0) n = (1.0 / S.d) * r;
        else { d3 o; perp_frame(e1, n, o); }
        e2 = cross(n, e1);
        const double c0[4] = {1.0, g - 1.0, -g, 0.0}, de[4] = {0.0, -1.0, 1.0, 0.0};
        S.cn = sqrt(dot4(c0, c0));
#pragma unroll
        for (int i = 0; i < 4; i++) S.c[i] = c0[i] / S.cn;
        orth4(de, S.c, nullptr, S.b2);
        const double k0 = dot4(de, S.c) * il, k1 = dot4(de, S.b2) * il, d2 = 2.0 * S.d * S.d, dc = -2.0 * S.d * S.cn;
        const double c2 = 2.0 * S.cn * S.cn;
        S.a[s5(0, 0)] = c2 - d2 * k0 * k0; S.a[s5(0, 1)] = -d2 * k0 * k1; S.a[s5(1, 1)] = -d2 * k1 * k1;
        S.a[s5(0, 3)] = dc * k0; S.a[s5(1, 3)] = dc * k1;
        S.a[s5(4, 4)] = c2;
    } else {
        const bool ee = type == T_EE;
        const d3 o = ee ? x[2] : x[1];
        const d3 w = x[0] - o, u = ee ? x[1] - x[0] : x[2] - o, v = x[3] - o;
        const d3 nn = cross(u, v);
        const double D2 = dot(nn, nn), D = sqrt(D2), iD = 1.0 / D;
        n = iD * nn;
        S.d = dot(w, n);
        const double al = dot(cross(w, v), nn) / D2, be = dot(cross(u, w), nn) / D2;
        const double lu = sqrt(dot(u, u)), ilu = 1.0 / lu;
        e1 = ilu * u;
        e2 = cross(n, e1);
        const double c0[4] = {ee ? 1.0 + al : 1.0, ee ? -al : al + be - 1.0, ee ? be - 1.0 : -al, -be};
        const double du[4] = {ee ? -1.0 : 0.0, ee ? 1.0 : -1.0, ee ? 0.0 : 1.0, 0.0};
        const double dv[4] = {0.0, ee ? 0.0 : -1.0, ee ? -1.0 : 0.0, 1.0};
        S.cn = sqrt(dot4(c0, c0));
#pragma unroll
        for (int i = 0; i < 4; i++) S.c[i] = c0[i] / S.cn;
        orth4(du, S.c, nullptr, S.b2);
        orth4(dv, S.c, S.b2, S.b3);
        // p = -(u* (du.x_n) + v* (dv.x_n)), u* = (v x n) / D, v* = (n x u) / D the dual basis
        const double u2 = dot(cross(v, n), e2) * iD, v2 = lu * iD;
        double p1[3], p2[3];
        const double ku[3] = {dot4(du, S.c), dot4(du, S.b2), 0.0};
        const double kv[3] = {dot4(dv, S.c), dot4(dv, S.b2), dot4(dv, S.b3)};
#pragma unroll
        for (int j = 0; j < 3; j++) { p1[j] = -ilu * ku[j]; p2[j] = -(u2 * ku[j] + v2 * kv[j]); }
        const double d2 = 2.0 * S.d * S.d, dc = 2.0 * S.d * S.cn;
#pragma unroll
        for (int i = 0; i < 3; i++) {
#pragma unroll
            for (int j = i; j < 3; j++) S.a[s5(i, j)] = -d2 * (p1[i] * p1[j] + p2[i] * p2[j]);
            S.a[s5(i, 3)] = dc * p1[i];
            S.a[s5(i, 4)] = dc * p2[i];
        }
        S.a[s5(0, 0)] += 2.0 * S.cn * S.cn;
    }
    store3(S.n, n); store3(S.e1, e1); store3(S.e2, e2);
}

// one rotation of the pair (P, Q): annihilates a_pq when it is above rounding
template <int P, int Q>
DV bool jacobi5_rotate(double (&a)[15], double (&v)[25], double floor2) {
    const double apq = a[s5(P, Q)], app = a[s5(P, P)], aqq = a[s5(Q, Q)];
    double c = 1.0, s = 0.0, t = 0.0;
    const bool rot = apq * apq > fmax(1e-30 * fabs(app * aqq), floor2);
    if (rot) {
        const double d = aqq - app, e = 2.0 * apq;
        const double h2 = fma(d, d, e * e);
        const double q = fabs(d) + h2 * rsqrt(h2);
        t = (d >= 0.0 ? e : -e) / q;
        c = rsqrt(fma(t, t, 1.0)); s = t * c;
        a[s5(P, P)] = app - t * apq;
        a[s5(Q, Q)] = aqq + t * apq;
        a[s5(P, Q)] = 0.0;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            if (k == P || k == Q) continue;
            const double kp = a[s5(k, P)], kq = a[s5(k, Q)];
            a[s5(k, P)] = c * kp - s * kq; a[s5(k, Q)] = s * kp + c * kq;
        }
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const double vp = v[5 * k + P], vq = v[5 * k + Q];
            v[5 * k + P] = c * vp - s * vq; v[5 * k + Q] = s * vp + c * vq;
        }
    }
    return rot;
}
// a <- V max(L, 0) V^T by cyclic Jacobi, disjoint pairs next to each other so
// that their rotations overlap; rotations below 1e-15 of their diagonal pair
// or 1e-14 of the matrix are skipped, and the sweeps end when all are
DV void psd_project5(double (&a)[15]) {
    double fro = 0.0, v[25];
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
        for (int j = i; j < 5; j++) fro += (i == j ? 1.0 : 2.0) * a[s5(i, j)] * a[s5(i, j)];
#pragma unroll
    for (int i = 0; i < 25; i++) v[i] = i % 6 == 0 ? 1.0 : 0.0;
    const double floor2 = 1e-28 * fro;
#pragma unroll 1
    for (int sweep = 0; sweep < 50; sweep++) {
        bool r = false;
        r |= jacobi5_rotate<0, 3>(a, v, floor2); r |= jacobi5_rotate<1, 4>(a, v, floor2);
        r |= jacobi5_rotate<0, 4>(a, v, floor2); r |= jacobi5_rotate<2, 3>(a, v, floor2);
        r |= jacobi5_rotate<0, 1>(a, v, floor2); r |= jacobi5_rotate<2, 4>(a, v, floor2);
        r |= jacobi5_rotate<1, 3>(a, v, floor2); r |= jacobi5_rotate<0, 2>(a, v, floor2);
        r |= jacobi5_rotate<1, 2>(a, v, floor2); r |= jacobi5_rotate<3, 4>(a, v, floor2);
        if (!r) break;
    }
    double l[5];
#pragma unroll
    for (int k = 0; k < 5; k++) l[k] = fmax(a[s5(k, k)], 0.0);
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
        for (int j = i; j < 5; j++) {
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < 5; k++) acc += l[k] * v[5 * i + k] * v[5 * j + k];
            a[s5(i, j)] = acc;
        }
}

// The contact's contribution to the Hessian in the five directions:
// projected mode, PSD(B1 f'' + B2 g g^T); reference mode (abd.py:247-251,
// :381-382), the line-line f'' alone projected, point-point without B1 f''.
DV void contact_matrix5(int type, bool projected, double B1, double B2, Stencil5& S) {
    const double gg = 4.0 * S.d * S.d * S.cn * S.cn;      // g g^T on the first direction
    if (projected) {
#pragma unroll
        for (int i = 0; i < 15; i++) S.a[i] *= B1;
        S.a[0] += B2 * gg;
        psd_project5(S.a);
    } else {
        if (type == T_EE) psd_project5(S.a);
        const double h = type == T_PP ? 0.0 : B1;
#pragma unroll
        for (int i = 0; i < 15; i++) S.a[i] *= h;
        S.a[0] += B2 * gg;
    }
}
