// search.cu — the line search of one Newton direction (gauss_newton.py:98-115)
// over the listed step (swept.cu): the CCD bound, the energies and the
// back-off, for every unit (scene or contact group) at once.
//
// A Newton iteration of a small scene is bound by the number of launches and
// by the latency of each, not by its bytes, so the search is three kernels:
//   k_ls_begin   the energy at the start, the CCD bound and the backup of the
//                body states in one pass over bodies, listed pairs and
//                vertices near a half-space; its last block sets the first
//                step lengths;
//   k_ls_apply   one trial's states and vertex positions (abd.py:768-785,
//                abd_simple.py:26-35), one warp per run of vertices of a body;
//                units that have accepted are left alone, so a batch whose
//                scenes have mostly converged costs only its live scenes;
//   k_ls_energy  the trial's energies; its last block accepts or halves.
// They replace thirteen launches before the search and eight per trial, each
// over every scene.  Per step: resting 16 x 16 net 11.85 -> 10.96 ms, 512
// uneven scenes (169 trials in two steps, most scenes converged after two
// iterations) 32.6 -> 22.1 ms, eight cubes 1.19 times faster.
#include "energy.cuh"
#include <algorithm>

// ------------------------------------------------------------------ shared pieces
// Body boxes of the listed step (bpair.cu), for skipping vertices that stay
// away from every half-space; null when the step was listed by the grid.
struct StepBoxes { const float4* lo; const float4* hi; };
// A body's swept box may reach a half-space: it comes within the barrier's
// distance or (ccd) holds a vertex whose distance may fall below ccd_scale times
// its present one.  A box that overflowed FP32 (a diverged increment) gives no
// distances and counts as near.
DV bool box_near_plane(float4 lo, float4 hi, const double* n, double dhat, bool ccd, double ccd_scale) {
    const double a0 = n[0] * lo.x, a1 = n[0] * hi.x, b0 = n[1] * lo.y, b1 = n[1] * hi.y, c0 = n[2] * lo.z, c1 = n[2] * hi.z;
    const double dmin = fmin(a0, a1) + fmin(b0, b1) + fmin(c0, c1) - n[3];
    const double dmax = fmax(a0, a1) + fmax(b0, b1) + fmax(c0, c1) - n[3];
    return !(dmin >= dhat) || (ccd && !(dmin >= ccd_scale * dmax));
}
// grid split over the three kinds of work; a warp looks at `group` chunks at
// once and then works on the live ones
struct LsGrid { int bodies, pairs, chunks, group; int total() const { return bodies + pairs + chunks; } };
// chunks a warp looks at: one while there are warps for every chunk, more in
// large batches, where most chunks belong to scenes that have converged
inline int chunk_group(int nchunks, int warps) { return std::min(32, std::max(1, (nchunks + warps - 1) / warps)); }

__global__ void k_ls_zero(int n, double* toi, double* e0, double* e0n, int ns, double* gg) {
    GS_LOOP(i, n) { toi[i] = 1.0; e0[i] = 0.0; e0n[i] = 0.0; }
    GS_LOOP(i, ns) gg[i] = 0.0;
}

struct LsArgs {
    int nb, ns, n; const int* n_dev;             // bodies, scenes, listed pairs (from the device when n_dev)
    const int4* list; const int4* chunks; int nchunks;
    Geo G; const double* p;                      // geometry at the current positions, displacement of the step
    const double* st; const double* J; double* backup;
    const double* g; const int* bscene; double* gg;   // gradient, and its squared norm per scene
    const int* unit; const int* skip;            // unit of a body; units left alone
    BodyTerms B; PairTerms T; StepBoxes box;
    int ccd; double ccd_scale; int ccd_it;
    double* E; double* En; double* toi;
};

// one role per block: bodies, then listed pairs, then vertices and half-spaces
template <bool BEGIN>
DV void ls_terms(const LsArgs& A, const LsGrid& g, int* capped) {
    const Geo& G = A.G;
    if ((int)blockIdx.x < g.bodies) {
        for (long base = (long)blockIdx.x * blockDim.x; base < A.nb; base += (long)g.bodies * blockDim.x) {
            const long b = base + threadIdx.x;
            bool valid = b < A.nb;
            const int u = valid ? A.unit[b] : 0;
            double e = 0, en = 0;
            if (valid) {
                const double* st = A.st + ST_STRIDE * b;
                if (BEGIN) {
#pragma unroll
                    for (int k = 0; k < 12; k++) A.backup[12 * b + k] = st[ST_NXT + k];
                }
                if (A.skip[u]) valid = false;
                else body_energy(st, G.mass[b], A.J[b], A.B, e, en);
            }
            warp_reduce_add(A.E, u, e, valid);
            warp_reduce_add(A.En, u, en, valid);
            if (BEGIN) {
                double n2 = 0;
                if (b < A.nb) {
#pragma unroll
                    for (int k = 0; k < 12; k++) n2 += A.g[12 * b + k] * A.g[12 * b + k];
                }
                warp_reduce_add(A.gg, b < A.nb ? A.bscene[b] : 0, n2, b < A.nb);
            }
        }
    } else if ((int)blockIdx.x < g.bodies + g.pairs) {
        const int n = A.n_dev ? *A.n_dev : A.n;
        for (long base = (long)(blockIdx.x - g.bodies) * blockDim.x; base < n; base += (long)g.pairs * blockDim.x) {
            const long c = base + threadIdx.x;
            bool valid = c < n;
            int u = 0;
            double e = 0, en = 0;
            if (valid) {
                const int4 C = A.list[c];
                const int2 ea = C.x == ABD_CONTACT_EE ? G.edges[C.y] : make_int2(C.y, C.y);
                u = A.unit[G.vbody[ea.x]];
                if (A.skip[u]) valid = false;
                else {
                    pair_energy(G, C, A.T, e, en);
                    if (BEGIN && A.ccd) {
                        int v[4];
                        if (C.x == ABD_CONTACT_EE) { const int2 eb = G.edges[C.z]; v[0] = ea.x; v[1] = ea.y; v[2] = eb.x; v[3] = eb.y; }
                        else { v[0] = C.y; v[1] = G.tris[3*C.z]; v[2] = G.tris[3*C.z+1]; v[3] = G.tris[3*C.z+2]; }
                        double xx[12], pp[12];
#pragma unroll
                        for (int k = 0; k < 4; k++)
#pragma unroll
                            for (int q = 0; q < 3; q++) { xx[3*k+q] = G.x[3*v[k]+q]; pp[3*k+q] = A.p[3*v[k]+q]; }
                        double t;
                        if (accd(C.x == ABD_CONTACT_EE ? 0 : 1, xx, pp, A.ccd_scale, 1.0, &t, capped, A.ccd_it)) atomic_min_pos(A.toi + u, t);
                    }
                }
            }
            warp_reduce_add(A.E, u, e, valid);
            warp_reduce_add(A.En, u, en, valid);
        }
    } else {
        const int lane = threadIdx.x & 31;
        const int w0 = ((blockIdx.x - g.bodies - g.pairs) * blockDim.x + threadIdx.x) >> 5;
        for (int w = w0 * g.group; w < A.nchunks; w += ((g.chunks * blockDim.x) >> 5) * g.group) {
            // the lanes look at one chunk each: its unit still searches, and
            // the body's swept box can reach a half-space
            int4 mine = make_int4(0, 0, 0, 0);
            bool live = false;
            if (lane < g.group && w + lane < A.nchunks) {
                mine = A.chunks[w + lane];              // body, first vertex, vertices, first chunk of the body
                if (!A.skip[A.unit[mine.x]]) {
                    const int s = G.bscene[mine.x];
                    for (int pl = G.sc_plane_begin[s]; pl < G.sc_plane_begin[s + 1] && !live; pl++) {
                        live = !A.box.lo || box_near_plane(A.box.lo[mine.x], A.box.hi[mine.x], G.planes + 4 * pl, A.T.dhat,
                                                           BEGIN && A.ccd, A.ccd_scale);
                    }
                }
            }
            for (unsigned m = __ballot_sync(0xffffffffu, live); m; m &= m - 1) {
                const int i = __ffs(m) - 1;
                const int4 c = make_int4(__shfl_sync(0xffffffffu, mine.x, i), __shfl_sync(0xffffffffu, mine.y, i),
                                         __shfl_sync(0xffffffffu, mine.z, i), 0);
                const int u = A.unit[c.x], s = G.bscene[c.x];
                double e = 0, en = 0, best = 1.0;
                for (int pl = G.sc_plane_begin[s]; pl < G.sc_plane_begin[s + 1]; pl++) {
                    const double* n = G.planes + 4 * pl;
                    for (int k = lane; k < c.z; k += 32) {
                        const int v = c.y + k;
                        plane_energy(G.x + 3L * v, n, A.T, e, en);
                        if (BEGIN && A.ccd) {
                            double d = n[0] * G.x[3*v] + n[1] * G.x[3*v+1] + n[2] * G.x[3*v+2] - n[3];
                            double vn = n[0] * A.p[3*v] + n[1] * A.p[3*v+1] + n[2] * A.p[3*v+2];
                            if (vn < 0) { double t = (1 - A.ccd_scale) * d / (-vn); if (t < 0) t = 0; if (t < best) best = t; }
                        }
                    }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    e += __shfl_xor_sync(0xffffffffu, e, o);
                    en += __shfl_xor_sync(0xffffffffu, en, o);
                    if (BEGIN) best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
                }
                if (lane == 0) {
                    atomicAdd(A.E + u, e);
                    atomicAdd(A.En + u, en);
                    if (BEGIN && best < 1.0) atomic_min_pos(A.toi + u, best);
                }
            }
        }
    }
}

// cap: the fraction of the increment the swept list covers (its CCD bound is
// a fraction of that shorter step)
__global__ void __launch_bounds__(256) k_ls_begin(LsArgs A, LsGrid g, int nu, const int* done, int* acc, double* alpha,
                                                  int* stall, double cap, Counters* cnt) {
    ls_terms<true>(A, g, &cnt->ccd_capped);
    if (!last_block(&cnt->ticket)) return;
    for (int s = threadIdx.x; s < nu; s += blockDim.x) {
        acc[s] = done[s];
        alpha[s] = (A.ccd ? fmin(1.0, __ldcg(A.toi + s)) : 1.0) * cap;
        if (!done[s]) stall[s] = 0;
    }
    if (threadIdx.x == 0) { cnt->ls_trials = 0; cnt->ls_nsw = A.n; }
}

// abd.py:768-785: nxt = backup - alpha du, and its vertices, for units not
// yet accepted; clears the trial's energy sums
__global__ void __launch_bounds__(256) k_ls_apply(int nchunks, int group, const int4* __restrict__ chunks, const double* __restrict__ backup,
        const double* __restrict__ du, const double* __restrict__ alpha, const int* __restrict__ skip,
        const int* __restrict__ unit, const double* __restrict__ xbar, double* __restrict__ st, double* __restrict__ x,
        float4* __restrict__ xf, int nu, double* e1, double* e1n) {
    GS_LOOP(i, nu) { e1[i] = 0.0; e1n[i] = 0.0; }
    const int lane = threadIdx.x & 31;
    for (int w = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * group; w < nchunks; w += ((gridDim.x * blockDim.x) >> 5) * group) {
        int4 mine = make_int4(0, 0, 0, 0);
        bool live = false;
        if (lane < group && w + lane < nchunks) { mine = chunks[w + lane]; live = !skip[unit[mine.x]]; }
        for (unsigned m = __ballot_sync(0xffffffffu, live); m; m &= m - 1) {
            const int i = __ffs(m) - 1;
            const int4 c = make_int4(__shfl_sync(0xffffffffu, mine.x, i), __shfl_sync(0xffffffffu, mine.y, i),
                                     __shfl_sync(0xffffffffu, mine.z, i), __shfl_sync(0xffffffffu, mine.w, i));
            const int u = unit[c.x];
            const double a = -alpha[u];
            double q[12];
    #pragma unroll
            for (int k = 0; k < 12; k++) q[k] = __fma_rn(a, du[12L * c.x + k], backup[12L * c.x + k]);
            if (c.w && lane < 12) {
                double v = q[0];
    #pragma unroll
                for (int k = 1; k < 12; k++) if (lane == k) v = q[k];
                st[(long)ST_STRIDE * c.x + ST_NXT + lane] = v;
            }
            for (int k = lane; k < c.z; k += 32) {
                const int v = c.y + k;
                const double x0 = xbar[3*v], x1 = xbar[3*v+1], x2 = xbar[3*v+2];
                double o[3];
    #pragma unroll
                for (int r = 0; r < 3; r++) {
                    double t = q[r];
                    t = __fma_rn(q[3 + r], x0, t);
                    t = __fma_rn(q[6 + r], x1, t);
                    t = __fma_rn(q[9 + r], x2, t);
                    o[r] = t;
                }
                x[3*v] = o[0]; x[3*v+1] = o[1]; x[3*v+2] = o[2];
                xf[v] = make_float4(__double2float_rn(o[0]), __double2float_rn(o[1]), __double2float_rn(o[2]), 0.f);
            }
        }
    }
}

// gauss_newton.py:107-113; an energy change within the FP64 evaluation error
// of the two energies (N0 + N1) is no increase.  MODE 0: energies only; 1: the
// decision; 2: the decision inside the line-search graph, whose while-node
// runs while units are pending, for at most LS_MAX_TRIALS trials
template <int MODE>
__global__ void __launch_bounds__(256) k_ls_energy(LsArgs A, LsGrid g, int nu, int* acc, double* alpha, const double* E0,
        const double* N0, double min_alpha, int* stall, Counters* cnt, cudaGraphConditionalHandle loop) {
    ls_terms<false>(A, g, nullptr);
    if (MODE == 0) return;
    if (!last_block(&cnt->ticket)) return;
    __shared__ int pending;
    if (threadIdx.x == 0) pending = 0;
    __syncthreads();
    for (int s = threadIdx.x; s < nu; s += blockDim.x) {
        if (acc[s]) continue;
        const double e0 = E0[s], e1 = __ldcg(A.E + s);
        if (e1 < e0 || e1 - e0 <= N0[s] + __ldcg(A.En + s)) acc[s] = 1;
        else if (alpha[s] * 0.5 < min_alpha) { acc[s] = 1; if (alpha[s] < ABD_LS_STALL_ALPHA) stall[s] = 1; }
        else { alpha[s] *= 0.5; atomicAdd(&pending, 1); }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        cnt->ls_pending = pending;
        if (MODE == 2) {
            const int t = cnt->ls_trials + 1;
            cnt->ls_trials = t;
            cudaGraphSetConditional(loop, (pending > 0 && t < LS_MAX_TRIALS) ? 1u : 0u);
        }
    }
}

// ------------------------------------------------------------------ host side
Geo eng_geo(Engine* E);

static LsArgs ls_args(Engine* E, const LsUnits& U, const int* skip, int slot) {
    LsArgs A;
    const AbdParams& P = E->P;
    A.nb = E->nb; A.ns = E->ns; A.n = E->n_sw; A.n_dev = nullptr;
    A.list = E->sw; A.chunks = E->vchunk; A.nchunks = E->nvchunk;
    A.G = eng_geo(E); A.p = E->pv; A.st = E->st; A.J = E->J; A.backup = E->backup;
    A.unit = U.bunit; A.skip = skip; A.B = body_terms(P); A.T = pair_terms(P);
    A.box = StepBoxes{nullptr, nullptr};
    eng_step_boxes(E, &A.box.lo, &A.box.hi);
    A.ccd = P.ccd; A.ccd_scale = P.ccd_scale; A.ccd_it = ccd_iters(P);
    A.E = U.d + slot * U.n; A.En = U.d + (slot == SD_E0 ? SD_E0N : SD_E1N) * U.n; A.toi = U.d + SD_TOI * U.n;
    return A;
}
// listed: pairs the grid is sized for (a graph keeps one size for every list)
static LsGrid ls_grid(const Engine* E, int threads, long listed) {
    auto blocks = [&](long n, int most) { return (int)std::min<long>((n + threads - 1) / threads, most); };
    LsGrid g;
    g.bodies = std::max(1, blocks(E->nb, NUM_SMS * 4));
    g.pairs = blocks(listed, NUM_SMS * 4);
    g.chunks = E->npl > 0 ? blocks(32L * E->nvchunk, NUM_SMS * 512 / threads) : 0;
    g.group = chunk_group(E->nvchunk, std::max(1, g.chunks * threads / 32));
    return g;
}

// start of a search along the listed step: CCD bound, start energies, backup
// of the states and the first step lengths
int eng_ls_begin(Engine* E, const LsUnits& U, const int* udone) {
    cudaStream_t s = E->stream;
    int rc = eng_transform(E);
    if (rc) return rc;
    LsArgs A = ls_args(E, U, udone, SD_E0);
    A.g = E->g; A.bscene = E->bscene; A.gg = E->scd + SD_GG * E->ns;
    k_ls_zero<<<grid_for(std::max(U.n, E->ns)), 256, 0, s>>>(U.n, A.toi, A.E, A.En, E->ns, A.gg);
    const int threads = TUNE_THREADS[tune_begin(E, TK_LIST_ENERGY, 3, 1)];
    const LsGrid g = ls_grid(E, threads, E->n_sw);
    k_ls_begin<<<g.total(), threads, 0, s>>>(A, g, U.n, udone, U.i + SI_ACC * U.n, U.d + SD_ALPHA * U.n, U.i + SI_STALL * U.n,
                                             E->sw_scale, E->dcnt);
    tune_end(E, TK_LIST_ENERGY);
    E->launches += 2;
    return ABD_OK;
}
// the states and positions of a trial at the units' step lengths
int eng_ls_apply(Engine* E, const LsUnits& U) {
    const int grid = (int)std::min<long>((32L * E->nvchunk + 255) / 256, NUM_SMS * 4);
    k_ls_apply<<<grid, 256, 0, E->stream>>>(E->nvchunk, chunk_group(E->nvchunk, grid * 8), E->vchunk, E->backup, E->du, U.d + SD_ALPHA * U.n,
        U.i + SI_ACC * U.n, U.bunit, E->xbar, E->st, E->x, E->xf, U.n, U.d + SD_E1 * U.n, U.d + SD_E1N * U.n);
    E->launches++;
    return ABD_OK;
}
// the trial's energies (decide 0), with the decision (1), or captured into the
// search graph (2, whose list length is read from the device)
int eng_ls_energy(Engine* E, const LsUnits& U, int decide, cudaGraphConditionalHandle loop) {
    int* acc = U.i + SI_ACC * U.n;
    LsArgs A = ls_args(E, U, acc, SD_E1);
    const int chosen = E->tune[TK_LIST_ENERGY].chosen;
    const int threads = TUNE_THREADS[chosen >= 0 ? chosen : 1];
    LsGrid g;
    if (decide == 2) { A.n_dev = &E->dcnt->ls_nsw; g = ls_grid(E, threads, (long)NUM_SMS * threads); }
    else g = ls_grid(E, threads, E->n_sw);
#define LS_ARGS A, g, U.n, acc, U.d + SD_ALPHA * U.n, U.d + SD_E0 * U.n, U.d + SD_E0N * U.n, E->P.ls_min_alpha, \
                U.i + SI_STALL * U.n, E->dcnt, loop
    if (decide == 0) k_ls_energy<0><<<g.total(), threads, 0, E->stream>>>(LS_ARGS);
    else if (decide == 1) k_ls_energy<1><<<g.total(), threads, 0, E->stream>>>(LS_ARGS);
    else k_ls_energy<2><<<g.total(), threads, 0, E->stream>>>(LS_ARGS);
#undef LS_ARGS
    E->launches++;
    return ABD_OK;
}
