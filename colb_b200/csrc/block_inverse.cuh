// block_inverse.cuh — inverse of a 12 x 12 body block by one warp.
#pragma once
#include "engine.cuh"

// Gauss-Jordan with partial pivoting on [D | I] in shared memory (M), lanes
// owning the 24 columns; V is column-major.  The inverse is left in
// M[..][12 ..]; false for a singular block.  All lanes call it.
template <class T>
DV bool block_inverse_warp(const T* V, double (*M)[25], int lane) {
    for (int e = lane; e < 288; e += 32) {
        int r = e / 24, c = e % 24;
        M[r][c] = c < 12 ? (double)V[c*12 + r] : (c - 12 == r ? 1.0 : 0.0);
    }
    __syncwarp();
    for (int c = 0; c < 12; c++) {
        // first row of largest magnitude in column c at or below the diagonal
        double best = lane >= c && lane < 12 ? fabs(M[lane][c]) : -1.0;
        int p = lane;
        for (int o = 16; o > 0; o >>= 1) {
            double ob = __shfl_xor_sync(0xffffffffu, best, o);
            int op = __shfl_xor_sync(0xffffffffu, p, o);
            if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
        }
        if (M[p][c] == 0.0) return false;
        if (p != c && lane < 24) { double t = M[p][lane]; M[p][lane] = M[c][lane]; M[c][lane] = t; }
        __syncwarp();
        double iv = 1.0 / M[c][c];
        __syncwarp();
        if (lane < 24) M[c][lane] *= iv;
        __syncwarp();
        double f[12];
#pragma unroll
        for (int r = 0; r < 12; r++) f[r] = M[r][c];
        __syncwarp();
        if (lane < 24) {
            double mc = M[c][lane];
#pragma unroll
            for (int r = 0; r < 12; r++)
                if (r != c && f[r] != 0.0) M[r][lane] -= f[r] * mc;
        }
        __syncwarp();
    }
    return true;
}
