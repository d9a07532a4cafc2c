// energy.cuh — per-item terms of the incremental potential and their FP64
// evaluation error, shared by the energy query (detect.cu, swept.cu) and the
// line search (search.cu).
#pragma once
#include "contact.cuh"

struct BodyTerms { double dt, g[3], k_ortho; };
struct PairTerms { int f32; double dhat; int barrier; double sc; };
inline BodyTerms body_terms(const AbdParams& P) {
    return BodyTerms{P.dt, {P.gravity[0], P.gravity[1], P.gravity[2]}, P.k_ortho};
}
inline PairTerms pair_terms(const AbdParams& P) { return PairTerms{P.ee_f32, P.dhat, P.barrier, P.kappa * P.dt * P.dt}; }

// inertia + orthogonality of one body (abd.py:53-66, ortho.py:9-20)
DV void body_energy(const double* st, double m, double J, const BodyTerms& T, double& e, double& en) {
    const double* now = st + ST_NOW; const double* nx = st + ST_NXT;
    const double dt = T.dt;
    double eo = ortho_energy(nx + ST_Q, T.k_ortho);
    double n0 = 0, n1 = 0, s0 = 0, s1 = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        double ct = now[ST_C+k] + dt * now[ST_V+k] + dt * dt * T.g[k];
        double d = nx[ST_C+k] - ct; n0 += d * d;
        s0 += fabs(d) * (fabs(nx[ST_C+k]) + fabs(ct));
    }
#pragma unroll
    for (int r = 0; r < 9; r++) {
        double qt = now[ST_Q+r] + dt * now[ST_QD+r];
        double d = nx[ST_Q+r] - qt; n1 += d * d;
        s1 += fabs(d) * (fabs(nx[ST_Q+r]) + fabs(qt));
    }
    e = eo * dt * dt + 0.5 * (n0 * m + n1 * J);
    en = (e + s0 * fabs(m) + s1 * fabs(J) + dt * dt * ortho_noise(nx + ST_Q, T.k_ortho)) * DBL_EPSILON;
}

// barrier of one listed pair; false when it is inactive
DV bool pair_energy(const Geo& G, int4 C, const PairTerms& T, double& e, double& en) {
    int4 stv; int type; double xb;
    if (!classify(G, C.x, C.y, C.z, T.f32, T.dhat, stv, type, xb)) return false;
    double b0, b1, b2; barrier3(T.barrier, xb, T.dhat * T.dhat, b0, b1, b2);
    e = b0 * T.sc;
    int vs[4] = {stv.x, stv.y, stv.z, stv.w};
    double L = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (vs[k] >= 0) L = fmax(L, fmax(fabs(G.x[3*vs[k]]), fmax(fabs(G.x[3*vs[k]+1]), fabs(G.x[3*vs[k]+2]))));
    // FP32 distances carry 2^29 times the FP64 rounding
    en = contact_noise(T.sc, b0, b1, xb, L, (T.f32 && C.x == ABD_CONTACT_EE) ? 536870912.0 : 1.0) * DBL_EPSILON;
    return true;
}

// barrier of one vertex against one half-space, added to e and en
DV void plane_energy(const double* x, const double* n, const PairTerms& T, double& e, double& en) {
    double d = n[0] * x[0] + n[1] * x[1] + n[2] * x[2] - n[3];
    if (!(d < T.dhat)) return;
    double L = fmax(fabs(x[0]), fmax(fabs(x[1]), fabs(x[2])));
    double b0, b1, b2; barrier3(T.barrier, d * d, T.dhat * T.dhat, b0, b1, b2);
    e += b0 * T.sc;
    en += contact_noise(T.sc, b0, b1, d * d, fmax(L, fabs(n[3])), 1.0) * DBL_EPSILON;
}
