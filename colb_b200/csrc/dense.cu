// dense.cu — direct solve of the Newton system (the reference's
// solver_config != "cg" branch, abd.py:637-654, which factors the assembled
// matrix with a cuSOLVER wrapper).
//
// The system decouples into the connected components of the body graph whose
// edges are the off-diagonal 12x12 blocks (two dynamic bodies joined by an
// active contact).  A component is factored on its own:
//   - one body: the inverse of its 12x12 block (k_du_scatter);
//   - Hessian projected to PSD and, in reverse Cuthill-McKee order, a body
//     bandwidth of at most BAND_WIDE: a banded L D L^T with the active window in
//     registers, all such components of bandwidth up to BAND_MAX in one launch
//     and the wider ones in another;
//   - otherwise (not projected, or a band solution that failed its check) up to
//     SMALL_MAX_BODIES bodies: one CTA per component factors it in shared
//     memory (blocked Cholesky by 12-wide body columns if projected; LU with
//     partial pivoting if not or when a pivot is not positive), all in one launch;
//   - larger components: the 12x12 blocks are scattered into a dense
//     column-major matrix and factored with cuSOLVER (Cholesky, or LU when
//     Cholesky reports a non-positive pivot).
// Mixed precision factors its FP32 blocks in FP64 on the band path, in FP32 on
// the others.  A band solution that could have met a small pivot is checked
// (band_check); where it fails, its component takes one of the last two paths in FP64.
#include "engine.cuh"
#include "block_inverse.cuh"
#include <cstring>
#include <cusolverDn.h>
#include <algorithm>

// Scatter the blocks of every body that belongs to a large component into
// that component's dense column-major matrix (16 lanes per body row).
template <class TV, class T>
__global__ void k_blocks_to_dense(int nb, const int* __restrict__ row_ptr, const int* __restrict__ bcol,
                                  const TV* __restrict__ vals, const int* __restrict__ bcomp,
                                  const int* __restrict__ blocal, const long long* __restrict__ comp_off,
                                  const long long* __restrict__ comp_n, int only_c, T* dense) {
    for (long base = (long)blockIdx.x * blockDim.x; base < (long)nb * 16; base += (long)gridDim.x * blockDim.x) {
        long t = base + threadIdx.x;
        int b = (int)(t / 16), l = (int)(t % 16);
        if (b >= nb || l >= 12) continue;
        int c = bcomp[b];
        if (c < 0 || (only_c >= 0 && c != only_c)) continue;
        long n = comp_n[c];
        T* A = dense + comp_off[c];
        long row = 12L * blocal[b] + l;
        for (int k = row_ptr[b]; k < row_ptr[b + 1]; k++) {
            long colb = 12L * blocal[bcol[k]];
            const TV* V = vals + (long)k * 144 + l;
#pragma unroll
            for (int j = 0; j < 12; j++) A[(colb + j) * n + row] = (T)V[j * 12];
        }
    }
}
// right-hand sides of large components, gathered in component order
template <class T>
__global__ void k_rhs_gather(int nb, const double* __restrict__ g, const int* __restrict__ bcomp,
                             const int* __restrict__ blocal, const long long* __restrict__ comp_rhs, T* x) {
    GS_LOOP(i, 12L * nb) {
        int b = (int)(i / 12), c = bcomp[b];
        if (c >= 0) x[comp_rhs[c] + 12L * blocal[b] + i % 12] = (T)g[i];
    }
}
// Neither the unpivoted factorization of a signed matrix nor one that replaced
// a pivot is backward stable: a small pivot grows without bound.  Every row of
// the band components that could meet one is therefore checked:
//   |g - A du|  <=  BAND_BACKWARD (|A| |du| + |g|) + |A - A^T| |du|
// A body with a row above that, or with a non-finite one, is marked in `bad`
// (pinned host memory; bad[nb]: any), and the host solves its component again
// with pivoting, in FP64 (eng_solve_again).  The bound is one FP32 rounding; a
// stable FP64 factorization is several orders below it (pivoted LU of nets in contact
// 1e-13 to 3e-10).  The last term is there because the factorization reads one
// entry of each symmetric pair, and FP32 blocks are symmetric only up to the
// order of their sums.  One warp per body (all lanes call it); its time is a few
// dependent loads, so the lanes look the transposed blocks up side by side.
constexpr double BAND_BACKWARD = 5.9604644775390625e-8;     // 2^-24
template <class T>
DV void band_check(int b, int nb, int lane, int* transposed, const int* __restrict__ row_ptr, const int* __restrict__ bcol,
                   const T* __restrict__ vals, const double* __restrict__ g, const double* __restrict__ du, int* bad) {
    const int l = lane % 12, h = lane / 12;                 // row, half of a block's columns
    double r = 0, s = 0, asym = 0;
    if (lane < 12) { r = g[12L * b + l]; s = fabs(r); }
    for (int k0 = row_ptr[b], k1 = row_ptr[b + 1]; k0 < k1; k0 += 32) {
        // (the pattern is symmetric: every transposed block is there)
        if (k0 + lane < k1) transposed[lane] = find_block(row_ptr, bcol, bcol[k0 + lane], b);
        __syncwarp();
        for (int k = k0; h < 2 && k < min(k0 + 32, k1); k++) {
            const T* V = vals + (long)k * 144 + 72 * h + l;
            const T* Vt = vals + (long)transposed[k - k0] * 144 + 12 * l + 6 * h;
            const double* x = du + 12L * bcol[k] + 6 * h;
#pragma unroll
            for (int j = 0; j < 6; j++) {
                const double a = V[j * 12], p = a * x[j];
                r -= p; s += fabs(p);
                asym += fabs((a - (double)Vt[j]) * x[j]);
            }
        }
        __syncwarp();
    }
    r += __shfl_sync(0xffffffffu, r, (lane + 12) & 31);
    s += __shfl_sync(0xffffffffu, s, (lane + 12) & 31);
    asym += __shfl_sync(0xffffffffu, asym, (lane + 12) & 31);
    if (lane < 12 && !(fabs(r) <= BAND_BACKWARD * s + asym && s <= DBL_MAX)) { bad[b] = 1; bad[nb] = 1; }
}

// du of every body, one warp each: large components from their dense solution, single
// bodies through the inverse of their 12x12 block; bodies of small
// components (bcomp -2) and band components (-3, -4) were written by
// k_small_solve / k_band_solve, and the former band components are checked
// (bad not null).  (The inverses of all bodies, single or not, in
// a launch of their own took 12 us for 256 bodies and 39 for 4,096.)
constexpr int DU_WARPS = 4;
template <class TV, class T>
__global__ void __launch_bounds__(32 * DU_WARPS) k_du_scatter(int nb, const double* __restrict__ g, const int* __restrict__ bcomp,
                             const int* __restrict__ blocal, const long long* __restrict__ comp_rhs,
                             const T* __restrict__ x, const int* __restrict__ row_ptr, const int* __restrict__ bcol,
                             const TV* __restrict__ vals, const int* __restrict__ bscene,
                             const int* __restrict__ ndone, double* du, int* bad) {
    __shared__ double sM[DU_WARPS][12][25];
    __shared__ int transposed[DU_WARPS][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double (*M)[25] = sM[w];
    for (int b = blockIdx.x * DU_WARPS + w; b < nb; b += gridDim.x * DU_WARPS) {
        const int c = bcomp[b];
        if (c == -3 && bad) { band_check<TV>(b, nb, lane, transposed[w], row_ptr, bcol, vals, g, du, bad); continue; }
        if (c <= -2 || ndone[bscene[b]]) continue;
        if (c >= 0) { if (lane < 12) du[12L * b + lane] = (double)x[comp_rhs[c] + 12L * blocal[b] + lane]; continue; }
        const int bi = find_block(row_ptr, bcol, b, b);
        const bool ok = block_inverse_warp<TV>(vals + (long)bi * 144, M, lane);
        if (lane < 12) {
            double acc = 0;
#pragma unroll
            for (int k = 0; k < 12; k++)
                acc += (double)(TV)(ok ? M[lane][12 + k] : (lane == k ? 1.0 : 0.0)) * g[12L * b + k];
            du[12L * b + lane] = acc;
        }
        __syncwarp();
    }
}

constexpr int SMALL_MAX_BODIES = 12;
constexpr int SMALL_THREADS = 256;

// Load the blocks of the component's bodies (local order sb[0..nbod)) into
// the row-major n x n matrix A (leading dimension ld) and g into x.
template <class TV, class T>
__device__ void small_fill(int nbod, int n, int ld, const int* sb, const int* __restrict__ blocal,
                           const int* __restrict__ row_ptr, const int* __restrict__ bcol, const TV* __restrict__ vals,
                           const double* __restrict__ g, T* A, T* x) {
    for (int e = threadIdx.x; e < n * ld; e += blockDim.x) A[e] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = warp; i < nbod; i += nw) {
        int b = sb[i];
        for (int k = row_ptr[b]; k < row_ptr[b + 1]; k++) {
            int j = blocal[bcol[k]];
            const TV* V = vals + (long)k * 144;
            for (int e = lane; e < 144; e += 32) {
                int cc = e / 12, r = e % 12;        // blocks are column-major
                A[(12 * i + r) * ld + 12 * j + cc] = (T)V[e];
            }
        }
        if (lane < 12) x[12 * i + lane] = (T)g[12L * b + lane];
    }
    __syncthreads();
}

// One CTA per small component: A du = g in shared memory.  status bit 0 is
// set when a component is singular (its du is zero).
template <class TV, class T>
__global__ void __launch_bounds__(SMALL_THREADS) k_small_solve(int nsmall, const int* __restrict__ sptr,
        const int* __restrict__ sbody, const int* __restrict__ blocal, const int* __restrict__ row_ptr,
        const int* __restrict__ bcol, const TV* __restrict__ vals, const double* __restrict__ g, int try_chol,
        double* du, int* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int flag, piv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int c = blockIdx.x; c < nsmall; c += gridDim.x) {
        const int* sb = sbody + sptr[c];
        const int nbod = sptr[c + 1] - sptr[c], n = 12 * nbod, ld = n + 1;
        T* A = (T*)smem_raw;
        T* x = A + n * ld;
        small_fill<TV, T>(nbod, n, ld, sb, blocal, row_ptr, bcol, vals, g, A, x);
        if (tid == 0) flag = try_chol ? 0 : 1;
        __syncthreads();
        // blocked right-looking Cholesky, lower triangle, 12-wide body columns;
        // flag is written by warp 0 in the diagonal step only and read right
        // after the barrier that follows it, so every thread takes the same branch
        for (int K = 0; try_chol && K < nbod; K++) {
            const int kb = 12 * K;
            if (warp == 0) {
                for (int j = 0; j < 12; j++) {
                    if (lane == 0) {
                        T d = A[(kb + j) * ld + kb + j];
                        if (!(d > (T)0)) flag = 1;
                        A[(kb + j) * ld + kb + j] = d > (T)0 ? sqrt(d) : (T)1;
                    }
                    __syncwarp();
                    T djj = A[(kb + j) * ld + kb + j];
                    if (lane > j && lane < 12) A[(kb + lane) * ld + kb + j] /= djj;
                    __syncwarp();
                    if (lane > j && lane < 12) {
                        T lij = A[(kb + lane) * ld + kb + j];
                        for (int cc = j + 1; cc <= lane; cc++) A[(kb + lane) * ld + kb + cc] -= lij * A[(kb + cc) * ld + kb + j];
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            if (flag) break;
            // panel: rows below solve L_ik D^T = A_ik
            for (int i = kb + 12 + tid; i < n; i += blockDim.x) {
                T* Ri = A + i * ld + kb;
                for (int j = 0; j < 12; j++) {
                    T a = Ri[j];
                    for (int t = 0; t < j; t++) a -= Ri[t] * A[(kb + j) * ld + kb + t];
                    Ri[j] = a / A[(kb + j) * ld + kb + j];
                }
            }
            __syncthreads();
            // trailing update of the lower triangle
            const int m = n - kb - 12;
            for (int e = tid; e < m * m; e += blockDim.x) {
                int i = kb + 12 + e / m, j = kb + 12 + e % m;
                if (j > i) continue;
                const T* Li = A + i * ld + kb;
                const T* Lj = A + j * ld + kb;
                T acc = 0;
#pragma unroll
                for (int t = 0; t < 12; t++) acc += Li[t] * Lj[t];
                A[i * ld + j] -= acc;
            }
            __syncthreads();
        }
        if (!flag) {
            // L y = g, then L^T du = y
            for (int K = 0; K < nbod; K++) {
                const int kb = 12 * K;
                if (tid == 0)
                    for (int j = 0; j < 12; j++) {
                        T a = x[kb + j];
                        for (int t = 0; t < j; t++) a -= A[(kb + j) * ld + kb + t] * x[kb + t];
                        x[kb + j] = a / A[(kb + j) * ld + kb + j];
                    }
                __syncthreads();
                for (int i = kb + 12 + tid; i < n; i += blockDim.x) {
                    T acc = 0;
                    for (int t = 0; t < 12; t++) acc += A[i * ld + kb + t] * x[kb + t];
                    x[i] -= acc;
                }
                __syncthreads();
            }
            for (int K = nbod - 1; K >= 0; K--) {
                const int kb = 12 * K;
                if (tid == 0)
                    for (int j = 11; j >= 0; j--) {
                        T a = x[kb + j];
                        for (int t = j + 1; t < 12; t++) a -= A[(kb + t) * ld + kb + j] * x[kb + t];
                        x[kb + j] = a / A[(kb + j) * ld + kb + j];
                    }
                __syncthreads();
                for (int i = tid; i < kb; i += blockDim.x) {
                    T acc = 0;
                    for (int t = 0; t < 12; t++) acc += A[(kb + t) * ld + i] * x[kb + t];
                    x[i] -= acc;
                }
                __syncthreads();
            }
        } else {
            // LU with partial pivoting on a fresh copy
            small_fill<TV, T>(nbod, n, ld, sb, blocal, row_ptr, bcol, vals, g, A, x);
            bool singular = false;
            for (int k = 0; k < n; k++) {
                if (warp == 0) {
                    T best = -1; int bi = k;
                    for (int i = k + lane; i < n; i += 32) {
                        T v = fabs(A[i * ld + k]);
                        if (v > best) { best = v; bi = i; }
                    }
                    for (int o = 16; o > 0; o >>= 1) {
                        T ob = __shfl_xor_sync(0xffffffffu, best, o);
                        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
                    }
                    if (lane == 0) piv = bi;
                }
                __syncthreads();
                const int p = piv;
                if (p != k) {
                    for (int j = tid; j < n; j += blockDim.x) { T t = A[k * ld + j]; A[k * ld + j] = A[p * ld + j]; A[p * ld + j] = t; }
                    if (tid == 0) { T t = x[k]; x[k] = x[p]; x[p] = t; }
                }
                __syncthreads();
                const T pv = A[k * ld + k];
                if (pv == (T)0) { singular = true; break; }
                for (int i = k + 1 + tid; i < n; i += blockDim.x) A[i * ld + k] /= pv;
                __syncthreads();
                const int m = n - k - 1;
                for (int e = tid; e < m * m; e += blockDim.x) {
                    int i = k + 1 + e / m, j = k + 1 + e % m;
                    A[i * ld + j] -= A[i * ld + k] * A[k * ld + j];
                }
                __syncthreads();
            }
            if (singular) {
                for (int i = tid; i < n; i += blockDim.x) x[i] = 0;
                if (tid == 0) atomicOr(status, 1);
                __syncthreads();
            } else {
                for (int k = 0; k < n; k++) {
                    const T xk = x[k];
                    for (int i = k + 1 + tid; i < n; i += blockDim.x) x[i] -= A[i * ld + k] * xk;
                    __syncthreads();
                }
                for (int k = n - 1; k >= 0; k--) {
                    if (tid == 0) x[k] /= A[k * ld + k];
                    __syncthreads();
                    const T xk = x[k];
                    for (int i = tid; i < k; i += blockDim.x) x[i] -= A[i * ld + k] * xk;
                    __syncthreads();
                }
            }
        }
        for (int i = tid; i < n; i += blockDim.x) du[12L * sb[i / 12] + i % 12] = (double)x[i];
        __syncthreads();
    }
}


// ------------------------------------------------------------------ band components
// 16-byte asynchronous global -> shared copies (cp.async, L1 bypassed): the
// band kernel fetches the next block row, right-hand side and backward factor
// column while it computes, so no global load latency sits on its critical
// path.  Addresses are 16-byte aligned (blocks of 144 doubles, 12-double rows).
DV void band_cp16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(sdst)), "l"(gsrc)
                 : "memory");
}
DV void band_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
DV void band_cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
DV void band_cp_wait_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
// named CTA barrier `id` over `n` threads (counted per thread, so a warp
// may reach it diverged): arrive only, which publishes this thread's earlier
// shared-memory writes to the waiting threads, or arrive and wait
DV void band_bar_arrive(int id, int n) { asm volatile("barrier.arrive %0, %1;" :: "r"(id), "r"(n) : "memory"); }
DV void band_bar_sync(int id, int n) { asm volatile("barrier.sync %0, %1;" :: "r"(id), "r"(n) : "memory"); }
// cluster barrier in two halves: arrive (release: this thread's earlier
// writes, global memory included, become visible to the cluster) and wait
// (acquire); every thread of the cluster arrives once per phase
DV void band_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
DV void band_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// A component whose bodies, in reverse Cuthill-McKee order, couple only
// bodies at most wb apart is a block band matrix: its factor A = L D L^T (L unit
// lower) has the same band.  A CTA factors it with the active window, the
// W = wb + 1 bodies that the current one couples, in registers.  Window thread
// (tr, tc) of a 12 x 12 grid owns entry (tr, tc) of every block (i, j), j <= i < W,
// of the window, whose slot i holds body k + i; after each body the window moves
// one block up and left (register moves), so every register index is a
// constant and the loop over bodies is short enough for the instruction
// caches.  Row threads own one or two window rows each: they eliminate.  Six
// pivots (half a body) take two barriers:
//   - the window threads have published the six pivot rows in shared memory;
//   - a row thread factors the 6 x 6 pivot block (every thread the same) and
//     eliminates its row's six entries, which gives the row's part of the
//     factor, the two vectors of the rank-6 update and its right-hand side's;
//   - the window threads publish the next pivot rows with that update applied,
//     and then apply it to their registers while the row threads go on.
// What bounds the kernel is this exchange, twice per body: each role waits for the
// other (barrier stall 4.6 per issue, FP64 pipe 14 % busy).  The pivots' own
// chain, a reciprocal of 74 cycles and two operations of 8 each, is about a
// seventh of it: 25 bodies one way, 300 pivots, 14 of 97 us for the first example
// below.  The right-hand side is one more column of the pivot
// rows.  After a body's pivots the row threads form
//   M_{k,d} = L_kk^-T L_{k+d,k}^T  and  a_k = L_kk^-T D^-1 y_k
// row by row (independent solves) and store them instead of the factor, so the
// backward recurrence x_k = a_k - sum_d M_{k,d} x_{k+d}, on one warp, is a short
// product per body, its records fetched four bodies at a time by the others.
// 46 bodies of bandwidth 5 take 97 us (a blocked Cholesky with the window in
// shared memory and one barrier per 12 x 12 factorization and product: 180),
// 20 of 3 43 us, 45 of 8 162, 61 of 9 201 (cuSOLVER's dense LDL^T, which
// took such a component before: 420), 92 of 11 363.
// PSD-projected FP64 matrices have positive pivots (one that is not sets bit 1
// of *status and is replaced by its magnitude).  SIGNED: mixed precision, whose
// FP32-rounded blocks can be indefinite (the 12-body blocks of a chain mail
// in contact have eigenvalues down to -2.9e3 of 1e9), factors them in FP64 with
// pivots of either sign, without exchanges; what a small pivot may have spoilt is
// found afterwards (band_check).
constexpr int BAND_MAX = 8;            // body bandwidths up to here: narrow kernel
constexpr int BAND_W = BAND_MAX + 1;   // its blocks per body
constexpr int BAND_WIDE = 11;          // up to here: wide kernel (78 window entries per thread)
constexpr int BAND_WTHREADS = 160;     // window threads: 12 x 12 in whole warps
constexpr int BAND_RTHREADS = 96;      // row threads: one row each up to 8 bodies, two rows in wider windows
constexpr int BAND_THREADS = BAND_WTHREADS + BAND_RTHREADS;
constexpr int BAND_ORD_MAX = 1024;     // bodies of a band component (order kept in shared memory)
constexpr int BAND_P = 6;              // pivots per step
constexpr int BAND_CHUNK = 4;          // bodies whose backward records are fetched at once
constexpr int band_ld(int w) { return 12 * w + 2; }            // a pivot row: columns, then its right-hand side
constexpr int band_ldr(int w) { return 12 * (w - 1) + 2; }     // a backward record's row: 12 wb entries of M, then a_k's
// dynamic shared memory in doubles for windows of at most bw bodies: two
// staged block rows, two chunks of backward records, the latest solution
// blocks, two sets of pivot rows and of the update's two vectors, the
// right-hand sides in passing, two L_kk, and the body order (ints)
constexpr int band_smem_doubles(int bw = BAND_W) {
    return (2 + 2 * BAND_CHUNK) * (bw * 144 + 12) + 16 * 12 + 6 * BAND_P * band_ld(bw) + 12 * bw + 288 + BAND_ORD_MAX / 2;
}
// a component of n bodies and body bandwidth wb is split between the two
// CTAs of its cluster at position m = (n - wb) / 2 when both halves keep at
// least wb / 2 + 6 block columns; -1 when it is factored by one CTA
inline int band_split_point(int n, int wb) { return n >= 2 * wb + 12 ? (n - wb) / 2 : -1; }


// Band blocks of every band component, contiguous and in FP64: A(i, i - d)
// of position i (component order), d = 0..bw - 1, row-major, at
// (loff + i bw + d); blocks outside the band or absent are zero.  One
// warp per block.
template <class TV>
__global__ void k_band_gather(int bw, int npos, const int* __restrict__ pcomp, const int* __restrict__ cptr,
                              const int* __restrict__ order, const int* __restrict__ cbw, const long long* __restrict__ loff,
                              const int* __restrict__ row_ptr, const int* __restrict__ bcol, const TV* __restrict__ vals,
                              double* Ab) {
    const int lane = threadIdx.x & 31;
    for (long item = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < (long)npos * bw;
         item += ((long)gridDim.x * blockDim.x) >> 5) {
        int p = (int)(item / bw), d = (int)(item % bw);
        int c = pcomp[p], i = p - cptr[c], j = i - d;
        if (d > cbw[c]) continue;                       // never read
        int bi = -1;
        if (j >= 0) bi = find_block(row_ptr, bcol, order[p], order[cptr[c] + j]);
        double* dst = Ab + (loff[c] + (long)i * bw + d) * 144;
        for (int e = lane; e < 144; e += 32) {
            int r = e / 12, cc = e % 12;
            dst[e] = bi >= 0 ? (double)vals[(long)bi * 144 + cc * 12 + r] : 0.0;     // row-major from column-major
        }
    }
}

// Warp-wide Cholesky factorization and inversion of 12 x 12 diagonal blocks
// would be a chain of 12 square roots and divisions per body; here the pivots
// are scalars, six divisions per step, which every row thread does for itself.

// What a CTA of k_band_solve works on: one sub-component in its own order.
struct BandJob {
    int N, wb, ncol1;                  // bodies, body bandwidth, bodies eliminated before the merge
    const double* A;                   // block A(i, i - d) at (i BW + d)
    double* L;                         // backward record of body k at (k BW) blocks
    double* Y;                         // right-hand sides of a handed-over separator at 12 k
    const int* ord;                    // bodies in order (shared memory)
    const double* g;
};
struct __align__(16) band_d2 { double x, y; };     // one 16-byte shared-memory access
struct BandSmem { double *stage, *cst, *xs, *rows, *pass, *lkk; int* ord; };
template <int BW>
DV BandSmem band_smem(unsigned char* raw) {
    BandSmem S;
    S.stage = (double*)raw;                                   // [2][BW * 144 + 12] (16-byte aligned for cp.async)
    S.cst = S.stage + 2 * (BW * 144 + 12);                    // [2][BAND_CHUNK][BW * 144 + 12]
    S.xs = S.cst + 2 * BAND_CHUNK * (BW * 144 + 12);          // [16][12]
    S.rows = S.xs + 16 * 12;                                  // [2] pivot rows, [2][2] update vectors, of BAND_P rows each
    S.pass = S.rows + 6 * BAND_P * band_ld(BW);               // [12 BW]
    S.lkk = S.pass + 12 * BW;                                 // [2][12][12]
    S.ord = (int*)(S.lkk + 288);                              // [BAND_ORD_MAX]
    return S;
}

// Shared memory of the elimination, and the pieces both roles use.  W: bodies of the window.
template <int W, int BW>
struct BandShared {
    static constexpr int LD = band_ld(W), M = 12 * W;         // right-hand side at column M
    const BandJob& J;
    const BandSmem& S;
    DV BandShared(const BandJob& j, const BandSmem& s) : J(j), S(s) {}
    DV double* pivots(int buf) const { return S.rows + buf * BAND_P * LD; }                  // P[BAND_P][LD]
    DV double* vec_c(int buf) const { return S.rows + (2 + 2 * buf) * BAND_P * LD; }         // c[row][BAND_P]: eliminated entries
    DV double* vec_t(int buf) const { return vec_c(buf) + BAND_P * LD; }                     // t[row][BAND_P]: the factor's
    DV const double* staged(int m) const { return S.stage + (m & 1) * (BW * 144 + 12); }
};

// Window threads (see above): the entries in registers.
template <int W, int BW>
struct BandWindow : BandShared<W, BW> {
    using B = BandShared<W, BW>;
    using B::LD; using B::J; using B::S; using B::pivots; using B::vec_c; using B::vec_t; using B::staged;
    static constexpr int off(int i, int j) { return i * (i + 1) / 2 + j; }
    double a[off(W, 0)];
    const int tid, tr, tc;
    DV BandWindow(const BandJob& j, const BandSmem& s)
        : BandShared<W, BW>(j, s), tid(threadIdx.x), tr(threadIdx.x / 12), tc(threadIdx.x % 12) {}
    DV bool owner() const { return tid < 144; }

    // block row m and its right-hand side into staging buffer m & 1
    DV void fetch_row(int m) const {
        double* dst = S.stage + (m & 1) * (BW * 144 + 12);
        const double* src = J.A + (long)m * BW * 144;
        for (int e = tid; e < W * 72 + 6; e += BAND_WTHREADS) {
            if (e < W * 72) band_cp16(dst + 2 * e, src + 2 * e);
            else { const int c = e - W * 72; band_cp16(dst + BW * 144 + 2 * c, J.g + 12L * J.ord[m] + 2 * c); }
        }
        band_cp_commit();
    }
    // the first W bodies
    DV void load() {
#pragma unroll
        for (int i = 0; i < W; i++)
#pragma unroll
            for (int j = 0; j <= i; j++) a[off(i, j)] = owner() ? J.A[((long)i * BW + i - j) * 144 + tid] : 0.0;
        if (W < J.N) fetch_row(W);
    }
    // window entry of block (i, j) with the update of vectors c, t applied
    template <int I, int JJ>
    DV double updated(const double* t, const double (&cv)[BAND_P]) const {
        const band_d2* tv = reinterpret_cast<const band_d2*>(t + (tr + 12 * I) * BAND_P);
        double v = a[off(I, JJ)], w = 0.0;
#pragma unroll
        for (int m = 0; m < BAND_P / 2; m++) {
            const band_d2 u = tv[m];
            v -= u.x * cv[2 * m];
            w -= u.y * cv[2 * m + 1];
        }
        return v + w;
    }
    // rows 6 .. 11 of slot 0 with the update applied; a pivot row's columns
    // are block (0, 0)'s row and, transposed, the blocks (i, 0) below it
    template <int I>
    DV void publish_half(double* P, const double* t, const double (&cv)[BAND_P]) const {
        if constexpr (I < W) {
            const double v = updated<I, 0>(t, cv);
            if (I == 0) { if (tr >= BAND_P) P[(tr - BAND_P) * LD + tc] = v; }
            else if (tc >= BAND_P) P[(tc - BAND_P) * LD + 12 * I + tr] = v;
            publish_half<I + 1>(P, t, cv);
        }
    }
    // rows 0 .. 5 of slot 1, which becomes slot 0, with the update applied
    template <int I>
    DV void publish_next(double* P, const double* t, const double (&cv)[BAND_P]) const {
        if constexpr (I < W) {
            const double v = updated<I, 1>(t, cv);
            if (I == 1) { if (tr < BAND_P) P[tr * LD + tc] = v; }
            else if (tc < BAND_P) P[tc * LD + 12 * (I - 1) + tr] = v;
            publish_next<I + 1>(P, t, cv);
        }
    }
    // the update of vectors `cb`
    DV void flush(int cb) {
        const band_d2* c = reinterpret_cast<const band_d2*>(vec_c(cb) + tc * BAND_P);
        const band_d2* t = reinterpret_cast<const band_d2*>(vec_t(cb) + tr * BAND_P);
#pragma unroll
        for (int m = 0; m < BAND_P / 2; m++) {
            band_d2 cv[W];
#pragma unroll
            for (int j = 0; j < W; j++) cv[j] = c[j * 6 * BAND_P + m];
#pragma unroll
            for (int i = 0; i < W; i++) {
                const band_d2 tv = t[i * 6 * BAND_P + m];
#pragma unroll
                for (int j = 0; j <= i; j++) { a[off(i, j)] -= tv.x * cv[j].x; a[off(i, j)] -= tv.y * cv[j].y; }
            }
        }
    }
    // eliminates bodies [k0, k1); before it slot i holds body k0 + i, after it body k1 + i
    DV void columns(int k0, int k1) {
        if (owner()) {
            double* P = pivots(0);
            if (tr < BAND_P) P[tr * LD + tc] = a[off(0, 0)];
#pragma unroll
            for (int i = 1; i < W; i++) if (tc < BAND_P) P[tc * LD + 12 * i + tr] = a[off(i, 0)];
        }
        band_bar_arrive(1, BAND_THREADS);                    // the first pivot rows are there
#pragma unroll 1
        for (int h = 2 * k0; h < 2 * k1; h++) {              // half bodies
            const int k = h >> 1, m = k + W, buf = h & 1;    // k0 may be odd: 2 k0 is even
            if (buf) band_cp_wait_all();                     // the entering body's row
            __syncthreads();                                 // the update's vectors (and that row) are there
            double* P = pivots(buf ^ 1);
            const double* t = vec_t(buf);
            const double* c = vec_c(buf) + (tc + (buf ? 12 : 0)) * BAND_P;
            const double* st = staged(m);
            const bool in = m < J.N;
            if (owner()) {
                double cv[BAND_P];
#pragma unroll
                for (int n = 0; n < BAND_P; n++) cv[n] = c[n];
                if (!buf) publish_half<0>(P, t, cv);
                else {
                    publish_next<1>(P, t, cv);
                    if (tc < BAND_P) P[tc * LD + 12 * (W - 1) + tr] = in ? st[(W - 1) * 144 + tid] : 0.0;
                }
            }
            if (h + 1 < 2 * k1) band_bar_arrive(1, BAND_THREADS);
            if (owner()) flush(buf);
            if (buf) {
                // one block up and left; body m enters below
#pragma unroll
                for (int i = 0; i + 1 < W; i++)
#pragma unroll
                    for (int j = 0; j <= i; j++) a[off(i, j)] = a[off(i + 1, j + 1)];
#pragma unroll
                for (int j = 0; j < W; j++) a[off(W - 1, j)] = in && owner() ? st[(W - 1 - j) * 144 + tid] : 0.0;
                if (m + 1 < J.N) fetch_row(m + 1);
            }
        }
        __syncthreads();
    }
    // the separator (bodies ncol1..N-1, slots 0..wb-1) into this sub-component's
    // unused record slots: block (p, q), p >= q, at (p BW + p - q), right-hand sides at Y + 12 p
    DV void hand_over() const {
        if (!owner()) return;
#pragma unroll
        for (int i = 0; i + 1 < W; i++)
#pragma unroll
            for (int j = 0; j <= i; j++) J.L[((long)(J.ncol1 + i) * BW + i - j) * 144 + tid] = a[off(i, j)];
    }
    // S = W0 + W1 - A_SS: adds the other CTA's separator (its blocks L1, right-hand
    // sides Y1; forward position i is its position nt1 - i, so its block (nt1 - j,
    // nt1 - i) is the transpose of block (i, j) here)
    DV void merge(const double* L1, const double*, int nt1) {
        if (!owner()) return;
        const int p0 = J.ncol1;
#pragma unroll
        for (int i = 0; i + 1 < W; i++)
#pragma unroll
            for (int j = 0; j <= i; j++)
                a[off(i, j)] += __ldcg(L1 + ((long)(nt1 - p0 - j) * BW + i - j) * 144 + tc * 12 + tr) -
                                J.A[((long)(p0 + i) * BW + i - j) * 144 + tid];
    }
};

// Row threads (see above): the elimination.
template <int W, int BW, bool SIGNED>
struct BandRows : BandShared<W, BW> {
    using B = BandShared<W, BW>;
    using B::LD; using B::M; using B::J; using B::S; using B::pivots; using B::vec_c; using B::vec_t; using B::staged;
    static constexpr int NR = 12 * W > BAND_RTHREADS ? 2 : 1; // rows of a thread: row, row + BAND_RTHREADS
    double rhs[NR];                      // right-hand sides of its rows
    int* status;
    const int row;
    DV BandRows(const BandJob& j, const BandSmem& s, int* st)
        : BandShared<W, BW>(j, s), status(st), row((int)threadIdx.x - BAND_WTHREADS) {}
    DV bool has_row(int n) const { return row + n * BAND_RTHREADS < 12 * W; }
    DV void load() {
#pragma unroll
        for (int n = 0; n < NR; n++) {
            const int r = row + n * BAND_RTHREADS;
            rhs[n] = has_row(n) ? J.g[12L * J.ord[r / 12] + r % 12] : 0.0;
        }
    }
    DV double pivot_inverse(double d) const {
        if (!SIGNED && !(d > 0.0)) { if (row == 0) atomicOr(status, 2); d = fabs(d) + 1e-30; }
        return 1.0 / d;
    }
    // rows of M_{k,d}, d >= 1, and a_k: entry n of row 12 (d - 1) + i at n LDR + row,
    // a_k's at n LDR + 12 wb (neighbouring threads write neighbouring places)
    DV void backward_record(int k, const double (&rec)[NR][12]) const {
        const double* lkk = S.lkk + (k & 1) * 144;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const int e = row + r * BAND_RTHREADS;
            if (!has_row(r) || (e > 0 && e < 12) || k + e / 12 >= J.N) continue;
            double v[12];
#pragma unroll
            for (int n = 0; n < 12; n++) v[n] = rec[r][n];
#pragma unroll
            for (int j = 11; j > 0; j--)
#pragma unroll
                for (int n = 0; n < j; n++) v[n] -= lkk[j * 12 + n] * v[j];
            double* o = J.L + (long)k * BW * 144 + (e == 0 ? 12 * (W - 1) : e - 12);
#pragma unroll
            for (int n = 0; n < 12; n++) o[n * band_ldr(W)] = v[n];
        }
    }
    DV void columns(int k0, int k1) {
        double rec[NR][12];              // the body's factor rows (thread 0, row 0: D^-1 y_k)
        if (row < BAND_P) pivots(0)[row * LD + M] = rhs[0];
#pragma unroll 1
        for (int h = 2 * k0; h < 2 * k1; h++) {
            const int k = h >> 1, buf = h & 1, q = buf * BAND_P;
            band_bar_sync(1, BAND_THREADS);
            const double* P = pivots(buf);
            double inv[BAND_P], l[BAND_P][BAND_P], y[BAND_P], c[NR][BAND_P];
            {
                double d[BAND_P][BAND_P];
#pragma unroll
                for (int n = 0; n < BAND_P; n++) {
#pragma unroll
                    for (int m = n; m < BAND_P; m++) d[m][n] = P[n * LD + q + m];
                    y[n] = P[n * LD + M];
#pragma unroll
                    for (int r = 0; r < NR; r++) c[r][n] = has_row(r) ? P[n * LD + row + r * BAND_RTHREADS] : 0.0;
                }
#pragma unroll
                for (int n = 0; n < BAND_P; n++) {
                    inv[n] = pivot_inverse(d[n][n]);
#pragma unroll
                    for (int m = n + 1; m < BAND_P; m++) l[m][n] = d[m][n] * inv[n];
#pragma unroll
                    for (int m = n + 1; m < BAND_P; m++) {
#pragma unroll
                        for (int o = n + 1; o <= m; o++) d[m][o] -= l[m][n] * d[o][n];
                        y[m] -= l[m][n] * y[n];
#pragma unroll
                        for (int r = 0; r < NR; r++) c[r][m] -= l[m][n] * c[r][n];
                    }
                }
            }
            double t[NR][BAND_P];
#pragma unroll
            for (int r = 0; r < NR; r++) {
                if (!has_row(r)) continue;
                const int e = row + r * BAND_RTHREADS;
                double r0 = rhs[r], r1 = 0.0;
#pragma unroll
                for (int n = 0; n < BAND_P; n++) {
                    t[r][n] = c[r][n] * inv[n];
                    vec_c(buf)[e * BAND_P + n] = c[r][n]; vec_t(buf)[e * BAND_P + n] = t[r][n];
                    if (n & 1) r1 -= t[r][n] * y[n]; else r0 -= t[r][n] * y[n];
                }
                rhs[r] = r0 + r1;
                // the next pivots' right-hand sides: rows 6 .. 11, or the next body's first six
                const int next = buf ? 12 : BAND_P;
                if (e >= next && e < next + BAND_P) pivots(buf ^ 1)[(e - next) * LD + M] = rhs[r];
                if (buf) S.pass[e] = rhs[r];
            }
            // L_kk for the solves
            if (row < 12) {
#pragma unroll
                for (int n = 0; n < BAND_P; n++) S.lkk[(k & 1) * 144 + row * 12 + q + n] = t[0][n];
            }
            __syncthreads();                                     // the update's vectors are there
            if (!buf) {
                // the window threads are publishing: the previous body's record
                if (k > k0) backward_record(k - 1, rec);
#pragma unroll
                for (int n = 0; n < BAND_P; n++)
#pragma unroll
                    for (int r = 0; r < NR; r++) rec[r][n] = r == 0 && row == 0 ? y[n] * inv[n] : t[r][n];
                continue;
            }
            // right-hand sides move up with the window
#pragma unroll
            for (int r = 0; r < NR; r++) {
#pragma unroll
                for (int n = 0; n < BAND_P; n++) rec[r][BAND_P + n] = r == 0 && row == 0 ? y[n] * inv[n] : t[r][n];
                if (!has_row(r)) continue;
                const int e = row + r * BAND_RTHREADS;
                rhs[r] = e < 12 * (W - 1) ? S.pass[e + 12] : (k + W < J.N ? staged(k + W)[BW * 144 + e - 12 * (W - 1)] : 0.0);
            }
        }
        if (k1 > k0) backward_record(k1 - 1, rec);
        __syncthreads();
    }
    DV void hand_over() const {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const int e = row + r * BAND_RTHREADS;
            if (e < 12 * (W - 1)) J.Y[12L * J.ncol1 + e] = rhs[r];
        }
    }
    DV void merge(const double*, const double* Y1, int nt1) {
        const int p0 = J.ncol1;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const int e = row + r * BAND_RTHREADS, p = p0 + e / 12;
            if (e < 12 * (W - 1)) rhs[r] += __ldcg(Y1 + 12L * (nt1 - p) + e % 12) - J.g[12L * J.ord[p] + e % 12];
        }
    }
};

// both roles' elimination of a sub-component; the roles meet at the same barriers
template <class Role>
DV void band_eliminate(Role& role, const BandJob& J, bool split, int crank, const double* L1, const double* Y1, int nt1) {
    role.load();
    // one loop, so that the elimination's code is there once
    int k0 = 0, k1 = J.ncol1;
#pragma unroll 1
    for (;;) {
        role.columns(k0, k1);
        if (!split || crank == 1 || k1 == J.N) break;
        band_cluster_arrive(); band_cluster_wait();       // CTA 1's half of S is in global memory
        role.merge(L1, Y1, nt1);
        k0 = k1; k1 = J.N;
    }
    if (split && crank == 1) role.hand_over();
}

// x_k = a_k - sum_d M_{k,d} x_{k+d} for k = kfirst down to klast, by warp 0, the
// solution blocks above kfirst already in xs (a ring of 16).  The records of
// BAND_CHUNK bodies are fetched at once by the other warps, one chunk ahead.
// Every thread calls it.
template <int W, int BW>
DV void band_backward(const BandJob& J, const BandSmem& S, int kfirst, int klast, double* du) {
    constexpr int LDR = band_ldr(W), REC = 12 * LDR;
    const int lane = threadIdx.x & 31;
    const bool solver = threadIdx.x < 32;
    if (kfirst < klast) return;
    // chunk q: bodies kfirst - q BAND_CHUNK and the BAND_CHUNK - 1 below it
    auto fetch = [&](int q) {
        for (int b = 0; b < BAND_CHUNK; b++) {
            const int k = kfirst - q * BAND_CHUNK - b;
            if (k < klast) break;
            double* dst = S.cst + ((q & 1) * BAND_CHUNK + b) * REC;
            const double* src = J.L + (long)k * BW * 144;
            for (int e = threadIdx.x - 32; e < REC / 2; e += BAND_THREADS - 32) band_cp16(dst + 2 * e, src + 2 * e);
        }
        band_cp_commit();
    };
    if (!solver) fetch(0);
    const int jj = lane % 12, hh = lane / 12;            // lanes jj and jj + 12 take half of each block's rows
    const int nq = (kfirst - klast) / BAND_CHUNK + 1;
#pragma unroll 1
    for (int q = 0; q < nq; q++) {
        if (!solver) {
            fetch(q + 1);                                // into the buffer chunk q - 1 used
            band_cp_wait_but_one();                      // chunk q
        }
        __syncthreads();                                 // chunk q is there
        if (solver) {
#pragma unroll 1
            for (int b = 0; b < BAND_CHUNK; b++) {
                const int k = kfirst - q * BAND_CHUNK - b;
                if (k < klast) break;
                const int nk = min(W - 1, J.N - 1 - k);
                double x = 0.0;
                if (lane < 24) {
                    const double* rec = S.cst + ((q & 1) * BAND_CHUNK + b) * REC + jj * LDR;
                    double acc[3] = {hh == 0 ? rec[12 * (W - 1)] : 0.0, 0.0, 0.0};
                    const band_d2* M = reinterpret_cast<const band_d2*>(rec + 6 * hh);
#pragma unroll
                    for (int d = 1; d < W; d++) {
                        if (d > nk) break;
                        const band_d2* xi = reinterpret_cast<const band_d2*>(S.xs + ((k + d) & 15) * 12 + 6 * hh);
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            const band_d2 u = M[(d - 1) * 6 + r], w = xi[r];
                            acc[r] = fma(-u.x, w.x, acc[r]);
                            acc[r] = fma(-u.y, w.y, acc[r]);
                        }
                    }
                    x = acc[0] + acc[1] + acc[2];
                }
                x += __shfl_sync(0xffffffffu, x, (lane + 12) & 31);
                if (lane < 12) { S.xs[(k & 15) * 12 + lane] = x; du[12L * J.ord[k] + lane] = x; }
                __syncwarp();
            }
        }
        __syncthreads();                                 // chunk q's buffer is free
    }
}

// One sub-component of a job on this CTA.  A job is a band component (ct)
// factored by CTA 0 alone, or a large one split in two: ct holds its
// bodies [0, m + wb) in order, cb the bodies [m, N) in reverse order, and
// S = [m, m + wb) separates [0, m) from [m + wb, N) (the band couples bodies
// at most wb apart).  CTA 0 eliminates [0, m) while CTA 1 eliminates
// [m + wb, N) from the far end; each leaves S in its window with its own
// Schur update applied.  After a cluster barrier CTA 0 adds CTA 1's update
// (S = W0 + W1 - A_SS, right-hand sides likewise), factors and solves S,
// and signals the solution at a second cluster barrier; then both CTAs run
// their backward halves.  The dependent chain shrinks from N bodies each
// way to about (N - wb) / 2 + wb.
// Not inlined, and its arguments by value: each width gets its own register
// allocation, and what the loops read stays in registers (46 bodies of
// bandwidth 5: 97 us, with all widths in one function 127).
template <int W, int BW, bool SIGNED>
__device__ __attribute__((noinline)) void band_job(BandJob J, bool split, int crank, const double* L1, const double* Y1,
                                                   int nt1, double* du, int* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const BandSmem S = band_smem<BW>(smem_raw);
    if ((int)threadIdx.x < BAND_WTHREADS) {
        BandWindow<W, BW> role(J, S);
        band_eliminate(role, J, split, crank, L1, Y1, nt1);
    } else {
        BandRows<W, BW, SIGNED> role(J, S, status);
        band_eliminate(role, J, split, crank, L1, Y1, nt1);
    }
    int first = J.N - 1;
    if (split && crank == 1) {
        __threadfence();
        band_cluster_arrive(); band_cluster_wait();       // S handed over
        band_cluster_arrive(); band_cluster_wait();       // S solved by CTA 0
        for (int e = threadIdx.x; e < J.wb * 12; e += BAND_THREADS) {
            const int p = J.ncol1 + e / 12;
            S.xs[(p & 15) * 12 + e % 12] = __ldcg(du + 12L * J.ord[p] + e % 12);
        }
        first = J.ncol1 - 1;
        __syncthreads();
    }
    int last = split && crank == 0 ? J.ncol1 : 0;
#pragma unroll 1
    for (;;) {
        band_backward<W, BW>(J, S, first, last, du);
        if (last == 0) break;
        __threadfence();
        band_cluster_arrive();                            // S solved
        first = last - 1; last = 0;
    }
    if (split && crank == 0) band_cluster_wait();
    if (!split) {
        band_cluster_arrive(); band_cluster_wait();
        band_cluster_arrive(); band_cluster_wait();
    }
}

// One job per cluster of two CTAs (band_job).  jobs holds (ct, cb, m) per
// job, cb = -1 for an unsplit component (m is then its size).  One CTA per SM
// (its registers allow no second).
template <int BW = BAND_W, bool SIGNED = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(BAND_THREADS, 1)
k_band_solve(int njobs, const int* __restrict__ jobs, const int* __restrict__ cptr,
        const int* __restrict__ order, const int* __restrict__ cbw, const long long* __restrict__ loff,
        const double* __restrict__ Ab, long long ltot, const double* __restrict__ g, double* Lg, double* du,
        int* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int* ord = band_smem<BW>(smem_raw).ord;
    const int tid = threadIdx.x;
    const int crank = blockIdx.x & 1;                         // rank in the cluster
    for (int jb = blockIdx.x >> 1; jb < njobs; jb += gridDim.x >> 1) {
        const int ct = jobs[3 * jb], cb = jobs[3 * jb + 1], msplit = jobs[3 * jb + 2];
        const bool split = cb >= 0;
        if (crank == 1 && !split) {
            // nothing to factor: keep the cluster barriers in step with CTA 0
            band_cluster_arrive(); band_cluster_wait();
            band_cluster_arrive(); band_cluster_wait();
            continue;
        }
        const int cc = crank == 0 ? ct : cb;
        BandJob J;
        J.N = cptr[cc + 1] - cptr[cc]; J.wb = cbw[cc];
        J.ncol1 = !split ? J.N : (crank == 0 ? msplit : J.N - J.wb);
        J.A = Ab + loff[cc] * 144;
        J.L = Lg + loff[cc] * 144;
        J.Y = Lg + ltot * 144 + (loff[cc] / BW) * 12;
        J.ord = ord; J.g = g;
        for (int e = tid; e < J.N; e += BAND_THREADS) ord[e] = order[cptr[cc] + e];
        __syncthreads();
        const double* L1 = split ? Lg + loff[cb] * 144 : nullptr;
        const double* Y1 = split ? Lg + ltot * 144 + (loff[cb] / BW) * 12 : nullptr;
        const int nt1 = split ? msplit + (cptr[cb + 1] - cptr[cb]) - 1 : 0;
#define BAND_CASE(w) case w: band_job<w, BW, SIGNED>(J, split, crank, L1, Y1, nt1, du, status); break
        if constexpr (BW == BAND_W) {
            switch (J.wb + 1) { BAND_CASE(2); BAND_CASE(3); BAND_CASE(4); BAND_CASE(5); BAND_CASE(6); BAND_CASE(7); BAND_CASE(8); BAND_CASE(9); }
        } else {
            switch (J.wb + 1) { BAND_CASE(10); BAND_CASE(11); BAND_CASE(12); }
        }
#undef BAND_CASE
        __syncthreads();
    }
}

struct DenseState {
    cusolverDnHandle_t h = nullptr;
    void* A = nullptr; size_t A_bytes = 0;
    void* rhs = nullptr; size_t rhs_bytes = 0;
    void* work = nullptr; size_t work_bytes = 0, work_es = 0; int work_n = 0;   // work_es: widest type it fits
    int* ipiv = nullptr;
    int* info = nullptr;                             // 2 per large component, from [2] on
    long long* comp_d = nullptr;                     // per large component: offset | rhs offset | n
    int* imap_d = nullptr; int* imap_h = nullptr;    // bmap | blocal | sptr | sbody | band maps | band factor offsets (blocks) | status
    void* Lg = nullptr; size_t Lg_bytes = 0;         // band factors
    void* Ab = nullptr;                              // band blocks gathered in component order (Lg_bytes)
    int* bad = nullptr;                              // pinned: bodies whose rows failed band_check, [nb]: any
    std::vector<unsigned long long> keys;
    std::vector<int> done, rp, col, act, parent, size, root, fill;
    std::vector<int> pos, members, mptr;
    bool smem_set[3] = {false, false, false};
    bool band_smem_set[2][2] = {};
};
static DenseState* ds_of(Engine* E) { return reinterpret_cast<DenseState*>(E->dense_state); }

constexpr int MAX_LARGE_COMPONENTS = 16;

void eng_dense_free(Engine* E) {
    DenseState* D = ds_of(E);
    if (!D) return;
    if (D->h) cusolverDnDestroy(D->h);
    void* ps[] = {D->A, D->rhs, D->work, D->ipiv, D->info, D->comp_d, D->imap_d, D->Lg, D->Ab};
    for (void* p : ps) if (p) cudaFree(p);
    if (D->imap_h) cudaFreeHost(D->imap_h);
    if (D->bad) cudaFreeHost(D->bad);
    delete D;
    E->dense_state = nullptr;
}

// bytes of the dense matrices if every scene were one component
long long eng_dense_bytes(Engine* E) {
    long long tot = 0;
    for (int s = 0; s < E->ns; s++) {
        long long n = 12LL * (E->h_body_begin[s + 1] - E->h_body_begin[s]);
        tot += n * n;
    }
    return tot * (E->mixed ? 4 : 8);
}

static int dense_init(Engine* E) {
    if (E->dense_state) return ABD_OK;
    DenseState* D = new DenseState();
    E->dense_state = D;
    auto fails = [&](const char* what) { eng_dense_free(E); return E->fail(ABD_ERR_CUDA, what); };
    if (cusolverDnCreate(&D->h) != CUSOLVER_STATUS_SUCCESS) return fails("cusolverDnCreate");
    cusolverDnSetStream(D->h, E->stream);
    // component maps, small-component lists, band sub-components (a split
    // component's separator appears in both halves) and band jobs
    size_t ni = 14 * (size_t)E->nb + 40;
    if (cudaMalloc(&D->imap_d, sizeof(int) * ni) != cudaSuccess) return fails("cudaMalloc maps");
    if (cudaMallocHost(&D->imap_h, sizeof(int) * ni) != cudaSuccess) return fails("cudaMallocHost maps");
    if (cudaMallocHost(&D->bad, sizeof(int) * (E->nb + 1)) != cudaSuccess) return fails("cudaMallocHost check flags");
    memset(D->bad, 0, sizeof(int) * (E->nb + 1));
    if (cudaMalloc(&D->info, sizeof(int) * (2 * MAX_LARGE_COMPONENTS + 2)) != cudaSuccess) return fails("cudaMalloc info");
    if (cudaMalloc(&D->comp_d, sizeof(long long) * 3 * MAX_LARGE_COMPONENTS) != cudaSuccess) return fails("cudaMalloc comps");
    return ABD_OK;
}

template <class T>
static int dense_reserve(Engine* E, DenseState* D, size_t a_elems, size_t rhs_elems, int nmax) {
    size_t es = sizeof(T);
    if (a_elems * es > D->A_bytes) {
        if (D->A) cudaFree(D->A);
        D->A_bytes = std::max(a_elems * es * 2, (size_t)1 << 20);
        if (cudaMalloc(&D->A, D->A_bytes) != cudaSuccess) { D->A = nullptr; D->A_bytes = 0; return E->fail(ABD_ERR_CUDA, "cudaMalloc dense matrices"); }
    }
    if (rhs_elems * es > D->rhs_bytes) {
        if (D->rhs) cudaFree(D->rhs);
        D->rhs_bytes = rhs_elems * es + 4096;
        if (cudaMalloc(&D->rhs, D->rhs_bytes) != cudaSuccess) { D->rhs = nullptr; D->rhs_bytes = 0; return E->fail(ABD_ERR_CUDA, "cudaMalloc dense rhs"); }
    }
    if (nmax > D->work_n || es > D->work_es) {
        // room for components up to twice this size (at most the whole handle)
        nmax = std::min(std::max(2 * nmax, 384), std::max(12 * E->nb, nmax));
        if (D->work) cudaFree(D->work);
        if (D->ipiv) cudaFree(D->ipiv);
        D->work = nullptr; D->ipiv = nullptr;
        D->work_es = std::max(es, D->work_es);
        size_t bytes = 0;
        int lw1 = 0, lw2 = 0;
        if (E->mixed) {
            cusolverDnSpotrf_bufferSize(D->h, CUBLAS_FILL_MODE_LOWER, nmax, (float*)D->A, nmax, &lw1);
            cusolverDnSgetrf_bufferSize(D->h, nmax, nmax, (float*)D->A, nmax, &lw2);
            bytes = ((size_t)std::max(lw1, lw2) + 32) * sizeof(float);
        }
        if (D->work_es == sizeof(double)) {
            cusolverDnDpotrf_bufferSize(D->h, CUBLAS_FILL_MODE_LOWER, nmax, (double*)D->A, nmax, &lw1);
            cusolverDnDgetrf_bufferSize(D->h, nmax, nmax, (double*)D->A, nmax, &lw2);
            bytes = std::max(bytes, ((size_t)std::max(lw1, lw2) + 32) * sizeof(double));
        }
        D->work_bytes = bytes;
        D->work_n = nmax;
        if (cudaMalloc(&D->work, D->work_bytes) != cudaSuccess || cudaMalloc(&D->ipiv, sizeof(int) * nmax) != cudaSuccess) {
            D->work_n = 0;
            return E->fail(ABD_ERR_CUDA, "cudaMalloc cusolver work");
        }
    }
    return ABD_OK;
}

template <class T>
static cusolverStatus_t potrf(DenseState* D, int n, T* A, T* work, int lwork, int* info) {
    if constexpr (sizeof(T) == 8) return cusolverDnDpotrf(D->h, CUBLAS_FILL_MODE_LOWER, n, A, n, work, lwork, info);
    else return cusolverDnSpotrf(D->h, CUBLAS_FILL_MODE_LOWER, n, A, n, work, lwork, info);
}
template <class T>
static cusolverStatus_t potrs(DenseState* D, int n, T* A, T* x, int* info) {
    if constexpr (sizeof(T) == 8) return cusolverDnDpotrs(D->h, CUBLAS_FILL_MODE_LOWER, n, 1, A, n, x, n, info);
    else return cusolverDnSpotrs(D->h, CUBLAS_FILL_MODE_LOWER, n, 1, A, n, x, n, info);
}
template <class T>
static cusolverStatus_t lu_solve(DenseState* D, int n, T* A, T* x, T* work, int* info) {
    cusolverStatus_t cs;
    if constexpr (sizeof(T) == 8) {
        cs = cusolverDnDgetrf(D->h, n, n, A, n, work, D->ipiv, info);
        if (cs == CUSOLVER_STATUS_SUCCESS) cs = cusolverDnDgetrs(D->h, CUBLAS_OP_N, n, 1, A, n, D->ipiv, x, n, info + 1);
    } else {
        cs = cusolverDnSgetrf(D->h, n, n, A, n, work, D->ipiv, info);
        if (cs == CUSOLVER_STATUS_SUCCESS) cs = cusolverDnSgetrs(D->h, CUBLAS_OP_N, n, 1, A, n, D->ipiv, x, n, info + 1);
    }
    return cs;
}

// Returns 1 in *fallback when there are more large components than
// MAX_LARGE_COMPONENTS or their matrices would exceed 4 GiB (the caller then
// runs the Krylov solver).  TV: the stored blocks, T: the arithmetic outside the
// band path.  again: the second solve of a system, in which the components that
// failed band_check take the pivoted paths.
template <class TV, class T>
static int dense_solve_t(Engine* E, int* iters, int* fallback, bool again) {
    *fallback = 0;
    int rc = eng_asm_wait(E);
    if (rc) return rc;
    if ((rc = dense_init(E))) return rc;
    DenseState* D = ds_of(E);
    std::vector<int> failed;
    if (again) failed.assign(D->bad, D->bad + E->nb);
    if (D->bad[E->nb]) memset(D->bad, 0, sizeof(int) * (E->nb + 1));
    cudaStream_t st = E->stream;
    const int* ndone = E->sci + SI_DONE * E->ns;
    const int nb = E->nb;
    // block pattern and done flags on the host (already there when the
    // assembly sent them): rows and columns, made from the keys where the
    // assembly sorted keys
    const int nk = E->nnzb_host;
    const int* rp; const int* col;
    const int* done;
    if (E->keys_host && E->row_bits) {
        rp = E->h_pattern; col = rp + nb + 1; done = E->h_done;
    } else {
        D->done.resize(E->ns);
        D->rp.assign(nb + 1, 0);
        D->col.resize(std::max(nk, 1));
        if (E->row_bits) {
            CUDA_TRY(cudaMemcpyAsync(D->rp.data(), E->row_ptr, sizeof(int) * (nb + 1), cudaMemcpyDeviceToHost, st));
            CUDA_TRY(cudaMemcpyAsync(D->col.data(), E->bcol, sizeof(int) * nk, cudaMemcpyDeviceToHost, st));
            CUDA_TRY(cudaMemcpyAsync(D->done.data(), ndone, sizeof(int) * E->ns, cudaMemcpyDeviceToHost, st));
            CUDA_TRY(eng_stream_sync(E));
        } else {
            D->keys.resize(std::max(nk, 1));
            if (E->keys_host && 2LL * nk <= E->h_pattern_cap) {
                if (nk > 0) memcpy(D->keys.data(), E->h_pattern, sizeof(unsigned long long) * nk);
                memcpy(D->done.data(), E->h_done, sizeof(int) * E->ns);
            } else {
                if (nk > 0) CUDA_TRY(cudaMemcpyAsync(D->keys.data(), E->ukeys, sizeof(unsigned long long) * nk, cudaMemcpyDeviceToHost, st));
                CUDA_TRY(cudaMemcpyAsync(D->done.data(), ndone, sizeof(int) * E->ns, cudaMemcpyDeviceToHost, st));
                CUDA_TRY(eng_stream_sync(E));
            }
            int m = 0;
            for (int k = 0; k < nk; k++) {           // sorted
                const unsigned long long key = D->keys[k];
                if (key == ~0ull) continue;
                D->rp[key / nb + 1]++;
                D->col[m++] = (int)(key % nb);
            }
            for (int b = 0; b < nb; b++) D->rp[b + 1] += D->rp[b];
        }
        rp = D->rp.data(); col = D->col.data(); done = D->done.data();
    }
    E->keys_host = false;
    // bodies coupled to others, of the scenes still iterating: all that the
    // analysis looks at (a batch has thousands of bodies that touch nothing)
    std::vector<int>& act = D->act;
    act.clear();
    for (int b = 0; b < nb; b++) if (rp[b + 1] - rp[b] > 1 && !done[E->h_bscene[b]]) act.push_back(b);
    // union-find, joined by off-diagonal blocks; a root is its component's first body
    std::vector<int>& parent = D->parent;
    parent.resize(nb); D->size.resize(nb); D->pos.resize(nb); D->root.resize(nb); D->mptr.resize(nb);
    for (int b : act) { parent[b] = b; D->size[b] = 0; D->pos[b] = -1; D->root[b] = -1; }
    auto find = [&](int x) { while (parent[x] != x) { parent[x] = parent[parent[x]]; x = parent[x]; } return x; };
    for (int r : act)
        for (int e = rp[r]; e < rp[r + 1] && col[e] < r; e++) {      // columns ascend, both directions are stored
            int a = find(r), b2 = find(col[e]);
            if (a != b2) { if (a < b2) parent[b2] = a; else parent[a] = b2; }
        }
    for (int b : act) D->size[find(b)]++;
    const bool projected = E->P.hess_mode == ABD_HESS_PROJECTED;
    // members of every component, ascending
    D->members.resize(std::max<size_t>(act.size(), 1));
    {
        int at = 0;
        for (int b : act) if (parent[b] == b) { D->mptr[b] = at; at += D->size[b]; D->size[b] = 0; }
        for (int b : act) { int r = find(b); D->members[D->mptr[r] + D->size[r]++] = b; }
    }
    // reverse Cuthill-McKee order of a component (BFS from a minimum-degree
    // body, neighbours by ascending degree, reversed) and its body bandwidth
    std::vector<int> nb_;
    auto rcm = [&](int r, std::vector<int>& out) {
        const int* m = D->members.data() + D->mptr[r];
        int n = D->size[r];
        auto degree = [&](int b) { return rp[b + 1] - rp[b]; };
        int start = m[0];
        for (int i = 1; i < n; i++) if (degree(m[i]) < degree(start)) start = m[i];
        out.clear(); out.push_back(start); D->pos[start] = 0;
        for (size_t h = 0; h < out.size(); h++) {
            int u = out[h];
            nb_.clear();
            for (int e = rp[u]; e < rp[u + 1]; e++) if (D->pos[col[e]] < 0) nb_.push_back(col[e]);
            std::sort(nb_.begin(), nb_.end(), [&](int a, int b) { return degree(a) != degree(b) ? degree(a) < degree(b) : a < b; });
            for (int v : nb_) if (D->pos[v] < 0) { D->pos[v] = 0; out.push_back(v); }
        }
        std::reverse(out.begin(), out.end());
        for (int i = 0; i < (int)out.size(); i++) D->pos[out[i]] = i;
        int bw = 0;
        for (int u : out)
            for (int e = rp[u]; e < rp[u + 1]; e++) bw = std::max(bw, std::abs(D->pos[u] - D->pos[col[e]]));
        return bw;
    };
    // components of scenes still iterating: band components (one CTA each,
    // Cholesky), small ones (one CTA each, dense in shared memory) and large
    // ones (cuSOLVER)
    int* h = D->imap_h;
    int* h_bmap = h; int* h_blocal = h + nb;
    std::fill_n(h_bmap, nb, -1);
    std::fill_n(h_blocal, nb, 0);
    std::vector<int> small_root, large_n, ord;
    std::vector<long long> large_off, large_rhs;
    long long aoff = 0, roff = 0;
    int nmax_large = 0, nmax_small = 0, small_bodies = 0, ncomp_band = 0, nsub = 0;
    // band components of the narrow and the wide kernel
    struct BandSet {
        int stride;                              // blocks per body
        std::vector<int> cptr{0}, bw, order, jobs;
        std::vector<long long> loff;
        long long blocks = 0;
    } sets[2] = {{BAND_W}, {BAND_WIDE + 1}};
    // a band sub-component: bodies in factor order, body bandwidth
    auto band_sub = [&](BandSet& B, const int* bodies, int len, int bw) {
        B.loff.push_back(B.blocks);
        B.blocks += (long long)len * B.stride;
        B.order.insert(B.order.end(), bodies, bodies + len);
        B.cptr.push_back((int)B.order.size());
        B.bw.push_back(bw);
        nsub++;
        return (int)B.bw.size() - 1;
    };
    std::vector<char> checked;                   // per band component
    auto has_failed = [&](int r) {
        const int* m = D->members.data() + D->mptr[r];
        for (int i = 0; i < D->size[r]; i++) if (failed[m[i]]) return true;
        return false;
    };
    for (int b : act) {
        int r = find(b), sz = D->size[r];
        // the band path takes every component of body bandwidth <= BAND_WIDE
        // of a projected Hessian, large ones split between the two CTAs of a
        // cluster; cuSOLVER takes wider ones, and the pivoted paths those that
        // failed the check of the band solution
        if (D->root[r] == -1 && projected && !(again && has_failed(r))) {
            int bw = rcm(r, ord);
            if (bw >= 1 && bw <= BAND_WIDE && sz <= BAND_ORD_MAX) {
                D->root[r] = -10 - ncomp_band++;          // marks a band component
                // FP64 of a narrow band replaces a pivot that is not positive and is not checked
                checked.push_back(sizeof(TV) == 4 || bw > BAND_MAX);
                BandSet& B = sets[bw > BAND_MAX];
                const int m = band_split_point(sz, bw);
                if (m > 0) {
                    // bodies [0, m + bw) forward, [m, sz) from the far end
                    const int ct = band_sub(B, ord.data(), m + bw, bw);
                    std::vector<int> rev(ord.rbegin(), ord.rend() - m);
                    const int cb = band_sub(B, rev.data(), sz - m, bw);
                    B.jobs.insert(B.jobs.end(), {ct, cb, m});
                } else {
                    const int ct = band_sub(B, ord.data(), sz, bw);
                    B.jobs.insert(B.jobs.end(), {ct, -1, sz});
                }
            }
        }
        if (D->root[r] <= -10) { h_bmap[b] = checked[-10 - D->root[r]] ? -3 : -4; continue; }
        if (D->root[r] < 0) {
            if (sz <= SMALL_MAX_BODIES) {
                D->root[r] = (int)small_root.size();
                small_root.push_back(r);
                nmax_small = std::max(nmax_small, 12 * sz);
            } else {
                if ((int)large_n.size() >= MAX_LARGE_COMPONENTS) { *fallback = 1; E->krylov_fallbacks++; return ABD_OK; }
                D->root[r] = (int)large_n.size();
                int n = 12 * sz;
                large_n.push_back(n); large_off.push_back(aoff); large_rhs.push_back(roff);
                aoff += (long long)n * n; roff += n;
                nmax_large = std::max(nmax_large, n);
            }
        }
        if (sz <= SMALL_MAX_BODIES) { h_bmap[b] = -2; small_bodies++; }
        else h_bmap[b] = D->root[r];
    }
    const int nsmall = (int)small_root.size(), nlarge = (int)large_n.size();
    E->comp_band += ncomp_band; E->comp_small += nsmall; E->comp_large += nlarge;

    if (aoff * (long long)sizeof(T) > (4LL << 30)) { *fallback = 1; E->krylov_fallbacks++; return ABD_OK; }
    // local body index inside its component (body order) and the small
    // components' body lists, packed into one upload
    int* h_sptr = h + 2 * nb; int* h_sbody = h_sptr + nsmall + 1;
    D->fill.assign(nsmall + nlarge, 0);
    h_sptr[0] = 0;
    for (int c = 0; c < nsmall; c++) h_sptr[c + 1] = h_sptr[c] + D->size[small_root[c]];
    for (int b : act) {
        int m = h_bmap[b];
        if (m == -2) {
            int c = D->root[find(b)];
            int l = D->fill[c]++;
            h_blocal[b] = l;
            h_sbody[h_sptr[c] + l] = b;
        } else if (m >= 0) {
            h_blocal[b] = D->fill[nsmall + m]++;
        }
    }
    // band components of each kernel: cptr | bandwidth | bodies in order |
    // component of each position | jobs, and the block offsets
    int* at = h_sbody + small_bodies;
    int* band_maps[2] = {nullptr, nullptr};
    for (int q = 0; q < 2; q++) {
        const BandSet& B = sets[q];
        band_maps[q] = at;
        auto put = [&](const std::vector<int>& v) { at = std::copy(v.begin(), v.end(), at); };
        put(B.cptr); put(B.bw); put(B.order);
        for (size_t c = 0; c < B.bw.size(); c++) at = std::fill_n(at, B.cptr[c + 1] - B.cptr[c], (int)c);
        put(B.jobs);
    }
    // the offsets behind them (8-byte aligned), and the status of the band and small kernels
    if ((at - h) & 1) *at++ = 0;
    const size_t loff_first = at - h;
    for (int q = 0; q < 2; q++)
        for (long long v : sets[q].loff) { memcpy(at, &v, sizeof v); at += 2; }
    *at = 0;
    int* d_status = D->imap_d + (at++ - h);
    const size_t nints = at - h;
    CUDA_TRY(cudaMemcpyAsync(D->imap_d, h, sizeof(int) * nints, cudaMemcpyHostToDevice, st));
    const int* d_bmap = D->imap_d; const int* d_blocal = D->imap_d + nb;
    const int* d_sptr = D->imap_d + 2 * nb; const int* d_sbody = d_sptr + nsmall + 1;
    if (nsub > 0) {
        size_t doubles[2];
        for (int q = 0; q < 2; q++) doubles[q] = (size_t)sets[q].blocks * 144 + 12 * sets[q].order.size();
        const size_t need = (doubles[0] + doubles[1]) * sizeof(double);
        if (need > D->Lg_bytes) {
            if (D->Lg) cudaFree(D->Lg);
            if (D->Ab) cudaFree(D->Ab);
            D->Lg = nullptr; D->Ab = nullptr;
            D->Lg_bytes = std::max(2 * need, (size_t)1 << 20);
            if (cudaMalloc(&D->Lg, D->Lg_bytes) != cudaSuccess || cudaMalloc(&D->Ab, D->Lg_bytes) != cudaSuccess) {
                D->Lg_bytes = 0;
                return E->fail(ABD_ERR_CUDA, "cudaMalloc band factors");
            }
        }
        int ph = phase_begin(E, PH_BAND);
        double bytes = 0;
        for (int q = 0; q < 2; q++) {
            const BandSet& B = sets[q];
            const int n = (int)B.bw.size(), npos = (int)B.order.size(), njobs = (int)B.jobs.size() / 3;
            if (n == 0) continue;
            const int* d_cptr = D->imap_d + (band_maps[q] - h);
            const int* d_bw = d_cptr + n + 1;
            const int* d_ord = d_bw + n;
            const int* d_pcomp = d_ord + npos;
            const int* d_jobs = d_pcomp + npos;
            const long long* d_loff = reinterpret_cast<const long long*>(D->imap_d + loff_first) + (q ? sets[0].bw.size() : 0);
            double* Ab = (double*)D->Ab + (q ? doubles[0] : 0);
            double* Lg = (double*)D->Lg + (q ? doubles[0] : 0);
            constexpr bool mixed = sizeof(TV) == 4;
            auto kernel = q ? k_band_solve<BAND_WIDE + 1, mixed> : k_band_solve<BAND_W, mixed>;
            const size_t smem = (size_t)band_smem_doubles(B.stride) * sizeof(double);
            if (!D->band_smem_set[q][mixed]) {
                CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                D->band_smem_set[q][mixed] = true;
            }
            k_band_gather<TV><<<grid_for(32L * npos * B.stride), 256, 0, st>>>(B.stride, npos, d_pcomp, d_cptr, d_ord, d_bw, d_loff,
                                                                             E->row_ptr, E->bcol, (const TV*)E->vals, Ab);
            // one cluster of two CTAs per job
            kernel<<<2 * njobs, BAND_THREADS, smem, st>>>(njobs, d_jobs, d_cptr, d_ord, d_bw, d_loff, Ab, B.blocks, E->g, Lg,
                                                          E->du, d_status);
            E->launches += 2;
            // per component: band blocks read, factor written and read back,
            // g read, y and du written and read
            for (int c = 0; c < n; c++)
                bytes += (B.cptr[c + 1] - B.cptr[c]) * ((B.bw[c] + 1) * 144.0 * sizeof(double) * 3 + 96.0 * 4);
        }
        phase_end(E, ph, bytes);
        if (!again && (E->P.test_inject & ABD_INJECT_BAND_CHECK)) {      // test hook: every band component fails
            for (int b : act) if (h_bmap[b] <= -3) D->bad[b] = 1;
            D->bad[nb] = 1;
        }
    }
    if (nsmall > 0) {
        size_t smem = ((size_t)nmax_small * (nmax_small + 1) + nmax_small) * sizeof(T);
        constexpr int attr = (sizeof(TV) == 8) + (sizeof(T) == 8);
        if (!D->smem_set[attr]) {
            const size_t nm = 12 * SMALL_MAX_BODIES;
            CUDA_TRY(cudaFuncSetAttribute(k_small_solve<TV, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)((nm * (nm + 1) + nm) * sizeof(T))));
            D->smem_set[attr] = true;
        }
        k_small_solve<TV, T><<<nsmall, SMALL_THREADS, smem, st>>>(nsmall, d_sptr, d_sbody, d_blocal, E->row_ptr, E->bcol,
                                                              (const TV*)E->vals, E->g, projected ? 1 : 0, E->du, d_status);
        E->launches++;
    }
    T* x = nullptr;
    if (nlarge > 0) {
        if ((rc = dense_reserve<T>(E, D, (size_t)aoff, (size_t)roff, nmax_large))) return rc;
        std::vector<long long> comp(3 * nlarge);
        for (int c = 0; c < nlarge; c++) { comp[c] = large_off[c]; comp[nlarge + c] = large_rhs[c]; comp[2 * nlarge + c] = large_n[c]; }
        CUDA_TRY(cudaMemcpyAsync(D->comp_d, comp.data(), sizeof(long long) * 3 * nlarge, cudaMemcpyHostToDevice, st));
        const long long* d_off = D->comp_d; const long long* d_rhs = D->comp_d + nlarge; const long long* d_n = D->comp_d + 2 * nlarge;
        T* A = (T*)D->A;
        x = (T*)D->rhs;
        CUDA_TRY(cudaMemsetAsync(A, 0, sizeof(T) * (size_t)aoff, st));
        k_blocks_to_dense<TV, T><<<grid_for(16L * nb), 256, 0, st>>>(nb, E->row_ptr, E->bcol, (const TV*)E->vals, d_bmap,
                                                                d_blocal, d_off, d_n, -1, A);
        k_rhs_gather<T><<<grid_for(12L * nb), 256, 0, st>>>(nb, E->g, d_bmap, d_blocal, d_rhs, x);
        E->launches += 2;
        T* work = (T*)D->work;
        int lwork = (int)(D->work_bytes / sizeof(T));
        std::vector<char> use_lu(nlarge, projected ? 0 : 1);
        if (projected) {
            for (int c = 0; c < nlarge; c++)
                if (potrf<T>(D, large_n[c], A + large_off[c], work, lwork, D->info + 2 + 2 * c) != CUSOLVER_STATUS_SUCCESS)
                    return E->fail(ABD_ERR_CUDA, "cusolver potrf");
            std::vector<int> info(2 * nlarge);
            CUDA_TRY(cudaMemcpyAsync(info.data(), D->info + 2, sizeof(int) * 2 * nlarge, cudaMemcpyDeviceToHost, st));
            CUDA_TRY(eng_stream_sync(E));
            for (int c = 0; c < nlarge; c++) {
                if (info[2 * c] != 0) {
                    // not positive definite after all: rebuild this component for LU
                    use_lu[c] = 1;
                    CUDA_TRY(cudaMemsetAsync(A + large_off[c], 0, sizeof(T) * (size_t)large_n[c] * large_n[c], st));
                    k_blocks_to_dense<TV, T><<<grid_for(16L * nb), 256, 0, st>>>(nb, E->row_ptr, E->bcol, (const TV*)E->vals, d_bmap,
                                                                            d_blocal, d_off, d_n, c, A);
                    E->launches++;
                } else if (potrs<T>(D, large_n[c], A + large_off[c], x + large_rhs[c], D->info + 3 + 2 * c) != CUSOLVER_STATUS_SUCCESS) {
                    return E->fail(ABD_ERR_CUDA, "cusolver potrs");
                }
            }
        }
        for (int c = 0; c < nlarge; c++)
            if (use_lu[c] && lu_solve<T>(D, large_n[c], A + large_off[c], x + large_rhs[c], work, D->info + 2 + 2 * c) != CUSOLVER_STATUS_SUCCESS)
                return E->fail(ABD_ERR_CUDA, "cusolver getrf/getrs");
    }
    k_du_scatter<TV, T><<<grid_for(32L * nb, 32 * DU_WARPS), 32 * DU_WARPS, 0, st>>>(nb, E->g, d_bmap, d_blocal,
        nlarge ? D->comp_d + nlarge : nullptr, x, E->row_ptr, E->bcol, (const TV*)E->vals, E->bscene, ndone, E->du, again ? nullptr : D->bad);
    E->launches++;
    *iters = 1;
    return ABD_OK;
}

int eng_solve_direct(Engine* E, int* iters, int* fallback, bool again) {
    if (E->mixed && !again) return dense_solve_t<float, float>(E, iters, fallback, false);
    if (E->mixed) return dense_solve_t<float, double>(E, iters, fallback, true);
    return dense_solve_t<double, double>(E, iters, fallback, again);
}
// after the host has waited for the last solve: a band solution failed its check
bool eng_solve_failed(const Engine* E) {
    const auto* D = reinterpret_cast<const DenseState*>(E->dense_state);
    return D && D->bad && *(volatile int*)(D->bad + E->nb);
}
