// block_inverse.cuh — inverse of a 12 x 12 body block by one warp.
#pragma once
#include "engine.cuh"

// Gauss-Jordan with partial pivoting on [D | I], lane j owning column j of the
// 24 in registers; V is column-major.  The inverse is left in M[..][12 ..];
// false for a singular block.  All lanes call it.  A column is a chain of one
// search, one division and one update; the lane that owns it searches its own
// registers and broadcasts, so nothing waits on shared memory: 6 us for a
// few blocks, 12 with the columns in shared memory.
template <class T>
DV bool block_inverse_warp(const T* V, double (*M)[25], int lane) {
    double a[12];
#pragma unroll
    for (int r = 0; r < 12; r++) a[r] = lane < 12 ? (double)V[lane * 12 + r] : (lane - 12 == r ? 1.0 : 0.0);
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 12; c++) {
        // first row of largest magnitude at or below the diagonal
        int p = c;
        double best = fabs(a[c]);
#pragma unroll
        for (int r = c + 1; r < 12; r++) if (fabs(a[r]) > best) { best = fabs(a[r]); p = r; }
        p = __shfl_sync(0xffffffffu, p, c);
#pragma unroll
        for (int r = c + 1; r < 12; r++) if (p == r) { const double t = a[r]; a[r] = a[c]; a[c] = t; }
        const double piv = __shfl_sync(0xffffffffu, a[c], c);
        ok = ok && piv != 0.0;
        const double iv = 1.0 / piv;
        a[c] *= iv;
#pragma unroll
        for (int r = 0; r < 12; r++) {
            if (r == c) continue;
            const double f = __shfl_sync(0xffffffffu, a[r], c);
            if (f != 0.0) a[r] -= f * a[c];
        }
    }
    if (lane >= 12 && lane < 24) {
#pragma unroll
        for (int r = 0; r < 12; r++) M[r][lane] = a[r];
    }
    __syncwarp();
    return ok;
}
