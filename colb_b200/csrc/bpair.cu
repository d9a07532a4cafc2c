// bpair.cu — three-level broad phase: bodies, then clusters of primitives of
// each overlapping body pair, then the primitives of each overlapping
// cluster pair.
//
// Affine bodies are rigid-ish meshes whose primitives are mostly surrounded
// by primitives of the same body, which never pair with them when
// self-contact is off.  A uniform grid over primitives therefore spends its
// time rejecting same-body neighbours.  Here:
//   1. one block per body forms the step's displacement and the swept,
//      padded box of every vertex and of the body;
//   2. one warp per body A tests A against every later body B of its scene
//      (and A against itself when self-contact is on) and appends the
//      overlapping pairs;
//   3. one block per body that has a pair forms the boxes of its clusters of
//      32 consecutive vertices, edges and triangles (neighbours in a mesh's
//      numbering are mostly neighbours in space), and one warp per body pair
//      and kind appends the overlapping cluster pairs;
//   4. one warp per cluster pair tests its (at most 32 x 32) primitive boxes
//      and runs the exact test on the overlapping ones, 32 at a time from a
//      queue, and appends hits;
//   5. hits are sorted by a 64-bit (kind, a, b) key, so the list comes out
//      in the same canonical order as the grid-based detection.
// Step 4 runs the reference's pair predicate (contact.py:158-168) in
// `detect` mode, or the Lipschitz reachability test along a step (see
// swept.cu) in `swept` mode.  Bodies must own contiguous vertex, edge and
// triangle ranges (as geometry.py:31-73 lays them out).
//
// What bounds it is the latency of dependent loads and the warp count, not
// bytes (7 MB of positions for a 16 x 16 net of 288-vertex links).  Staging
// all primitives of both bodies of a pair in one block, as an earlier form
// of step 4 did, forms every primitive box once per body pair (14 times more
// boxes than step 3 on that net) and leaves most of the block idle in the
// narrow tests; the figures are at bp_build.
#include "contact.cuh"
#include <cub/cub.cuh>
#include <climits>
#include <cstring>

Geo eng_geo(Engine* E);
int eng_grow_swept(Engine* E, int need);
int eng_grow_contacts(Engine* E, int need);
int eng_pg_candidates(Engine* E, double filt);

#define BP_CL 32            // primitives of a cluster: one per lane

DV float4 fmin4(float4 a, float4 b) { return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.f); }
DV float4 fmax4(float4 a, float4 b) { return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.f); }
DV bool overlap(float4 al, float4 ah, float4 bl, float4 bh) {
    return !(al.x > bh.x || ah.x < bl.x || al.y > bh.y || ah.y < bl.y || al.z > bh.z || ah.z < bl.z);
}

// swept (x .. x+p) padded box of one vertex, outward rounded
DV void vbox(const double* x, const double* p, float pad, float4& lo, float4& hi) {
    double a0 = x[0], a1 = x[1], a2 = x[2];
    double b0 = a0 + p[0], b1 = a1 + p[1], b2 = a2 + p[2];
    lo = make_float4(__fsub_rd(__double2float_rd(fmin(a0, b0)), pad), __fsub_rd(__double2float_rd(fmin(a1, b1)), pad),
                     __fsub_rd(__double2float_rd(fmin(a2, b2)), pad), 0.f);
    hi = make_float4(__fadd_ru(__double2float_ru(fmax(a0, b0)), pad), __fadd_ru(__double2float_ru(fmax(a1, b1)), pad),
                     __fadd_ru(__double2float_ru(fmax(a2, b2)), pad), 0.f);
}

// body boxes alone, one warp per body: the contact groups form their own, for
// steps listed by the grid as well as by step 1
__global__ void k_body_boxes(int nb, const int* __restrict__ vbeg, const double* __restrict__ x, const double* __restrict__ p,
                             float pad, float4* blo, float4* bhi) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    for (int b = warp; b < nb; b += (gridDim.x * blockDim.x) >> 5) {
        float4 lo = make_float4(3e38f, 3e38f, 3e38f, 0.f), hi = make_float4(-3e38f, -3e38f, -3e38f, 0.f);
        for (int v = vbeg[b] + lane; v < vbeg[b+1]; v += 32) {
            float4 l, h; vbox(x + 3L * v, p + 3L * v, pad, l, h);
            lo = fmin4(lo, l); hi = fmax4(hi, h);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o)); lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
            lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o)); hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
            hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o)); hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
        }
        if (lane == 0) { blo[b] = lo; bhi[b] = hi; }
    }
}

// 2. body pairs (a <= b, same scene); a == b only with self-contact
__global__ void k_body_pairs(int nb, const int* __restrict__ bscene, const int* __restrict__ sc_body_begin,
                             const float4* __restrict__ blo, const float4* __restrict__ bhi, int self_contact,
                             int2* out, int cap, int* count, int* paired) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    for (int a = warp; a < nb; a += (gridDim.x * blockDim.x) >> 5) {
        int s = bscene[a];
        int end = sc_body_begin[s + 1];
        float4 al = blo[a], ah = bhi[a];
        for (int b = a + (self_contact ? 0 : 1) + lane; b < end; b += 32) {
            if (!overlap(al, ah, blo[b], bhi[b])) continue;
            int at = atomicAdd(count, 1);
            if ((unsigned)at < (unsigned)cap) out[at] = make_int2(a, b);
            paired[a] = 1; paired[b] = 1;
        }
    }
}

struct BpArgs {
    Geo G; const float* pmag;
    const float4* vlo; const float4* vhi;          // per-vertex swept boxes of this build
    double lim; double filt; int mode;              // mode 0 swept (Lipschitz, lim), 1 detect (predicate, filt)
    int f32;
    unsigned long long* out; int cap; int* count;
};

DV bool bp_ee_ok(const BpArgs& A, int i, int j) {
    const Geo& G = A.G;
    int2 a = G.edges[i], b = G.edges[j];
    if (a.x == b.x || a.x == b.y || a.y == b.x || a.y == b.y) return false;
    if (A.mode == 1) { double s, t, d; return ee_test(G, i, j, A.f32, 1, A.filt, s, t, d); }
    double s, t, d;
    seg_seg_f64(G.x + 3*a.x, G.x + 3*a.y, G.x + 3*b.x, G.x + 3*b.y, 1e-12, s, t, d);
    double L = (double)fmaxf(A.pmag[a.x], A.pmag[a.y]) + (double)fmaxf(A.pmag[b.x], A.pmag[b.y]);
    return d - L < A.lim;
}
DV bool bp_pt_ok(const BpArgs& A, int pv, int t) {
    const Geo& G = A.G;
    int a = G.tris[3*t], b = G.tris[3*t+1], c = G.tris[3*t+2];
    if (pv == a || pv == b || pv == c) return false;
    if (A.mode == 1) return pt_test(G, pv, t, 1, A.filt);
    double d = sqrt(pt_dist2(G.x + 3*pv, G.x + 3*a, G.x + 3*b, G.x + 3*c));
    double L = (double)A.pmag[pv] + (double)fmaxf(A.pmag[a], fmaxf(A.pmag[b], A.pmag[c]));
    return d - L < A.lim;
}
// the hit counter stops growing once it has passed the capacity (by at most
// the threads in flight), so a pathological step (a displacement that makes every
// primitive pair reachable) cannot wrap it; the host then grows the buffer a
// bounded number of times and reports ABD_ERR_CONTACT_OVERFLOW.  A counter that
// only equals the capacity still counts: the first hit without a place must
// show, or the host would take a list that lacks it for complete.
DV void bp_emit(const BpArgs& A, int kind, int a, int b) {
    if (*(volatile int*)A.count > A.cap) return;
    int at = atomicAdd(A.count, 1);
    if ((unsigned)at < (unsigned)A.cap) A.out[at] = ((unsigned long long)kind << 62) | ((unsigned long long)a << 31) | (unsigned long long)b;
}

// ---- step 1: displacements and boxes
// Clusters of body b start at beg[b] / 32 + b: with at most ceil(n / 32) of
// them per body the ranges of successive bodies never overlap, so no table
// is needed.
DV int cl_first(const int* beg, int b) { return (beg[b] >> 5) + b; }
DV int cl_count(const int* beg, int b) { return (beg[b + 1] - beg[b] + BP_CL - 1) >> 5; }
// float <-> int with the same order, for the integer warp reductions
DV int f_ord(float f) { int i = __float_as_int(f); return i ^ ((i >> 31) & 0x7fffffff); }
DV float f_unord(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }
// union of the lanes' boxes in every lane (a lane without one passes an
// empty box); NaN bounds are ignored, as fminf / fmaxf do
DV void warp_union(float4& lo, float4& hi) {
    const unsigned full = 0xffffffffu;
    lo.x = f_unord(__reduce_min_sync(full, f_ord(fminf(lo.x, 3e38f)))); lo.y = f_unord(__reduce_min_sync(full, f_ord(fminf(lo.y, 3e38f))));
    lo.z = f_unord(__reduce_min_sync(full, f_ord(fminf(lo.z, 3e38f)))); hi.x = f_unord(__reduce_max_sync(full, f_ord(fmaxf(hi.x, -3e38f))));
    hi.y = f_unord(__reduce_max_sync(full, f_ord(fmaxf(hi.y, -3e38f)))); hi.z = f_unord(__reduce_max_sync(full, f_ord(fmaxf(hi.z, -3e38f))));
}
DV void empty_box(float4& lo, float4& hi) { lo = make_float4(3e38f, 3e38f, 3e38f, 0.f); hi = make_float4(-3e38f, -3e38f, -3e38f, 0.f); }

struct BpBoxes {
    float4 *vlo, *vhi, *blo, *bhi, *cl[3], *ch[3];   // clusters of vertices, edges, triangles
    int* still;                                      // the body did not move in the swept build that wrote its boxes
    int* paired;                                     // the body is in a body pair of this build
    int* clok;                                       // its cluster boxes belong to its present vertex boxes
};
struct BpDisp {                                                      // dq null: static positions
    const double* dq; double sign; const double* xbar; const double* mass; const int* bscene; const int* done;
    double* pv; float* pmag;
};
constexpr int BOX_THREADS = 128;
__global__ void __launch_bounds__(BOX_THREADS) k_bp_boxes(int nb, const int* __restrict__ vbeg, const double* __restrict__ x,
        BpDisp D, float pad, int keep, BpBoxes B, int* cnt) {
    if (blockIdx.x == 0 && threadIdx.x < 8) cnt[threadIdx.x] = 0;         // the build's counts
    __shared__ float4 slo[BOX_THREADS / 32], shi[BOX_THREADS / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        double d[12];
        bool dyn = false;
        if (threadIdx.x == 0) B.paired[b] = 0;
        if (D.dq) {
            dyn = D.mass[b] > 0.0 && !D.done[D.bscene[b]];
            // pinned, or its scene has converged: the boxes of the last
            // build, in which it did not move either, are still its boxes
            if (!dyn && keep && B.still[b]) continue;
            if (dyn) {
#pragma unroll
                for (int k = 0; k < 12; k++) d[k] = D.dq[12L * b + k];
            }
        }
        float4 rlo, rhi;
        empty_box(rlo, rhi);
        for (int v = vbeg[b] + threadIdx.x, v1 = vbeg[b + 1]; v < v1; v += BOX_THREADS) {
            double q[3] = {0.0, 0.0, 0.0};
            if (D.dq) {
                if (dyn) {
                    const double x0 = D.xbar[3*v], x1 = D.xbar[3*v+1], x2 = D.xbar[3*v+2];
#pragma unroll
                    for (int k = 0; k < 3; k++) q[k] = D.sign * (d[k] + x0 * d[3+k] + x1 * d[6+k] + x2 * d[9+k]);
                }
                D.pv[3*v] = q[0]; D.pv[3*v+1] = q[1]; D.pv[3*v+2] = q[2];
                D.pmag[v] = __double2float_ru(sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]));
            }
            float4 l, h;
            vbox(x + 3L * v, q, pad, l, h);
            B.vlo[v] = l; B.vhi[v] = h;
            rlo = fmin4(rlo, l); rhi = fmax4(rhi, h);
        }
        warp_union(rlo, rhi);
        if (lane == 0) { slo[warp] = rlo; shi[warp] = rhi; }
        __syncthreads();           // everyone has read the body's flag
        if (threadIdx.x == 0) {
            for (int w = 1; w < BOX_THREADS / 32; w++) { rlo = fmin4(rlo, slo[w]); rhi = fmax4(rhi, shi[w]); }
            B.blo[b] = rlo; B.bhi[b] = rhi;
            B.still[b] = !dyn;
            B.clok[b] = 0;
        }
        __syncthreads();           // slo / shi are read before the next body writes them
    }
}

// ---- step 3: cluster boxes of the bodies that have a pair
__global__ void __launch_bounds__(BOX_THREADS) k_bp_clboxes(int nb, const int* __restrict__ vbeg, const int* __restrict__ ebeg,
        const int* __restrict__ tbeg, const int2* __restrict__ edges, const int* __restrict__ tris, int do_ee, int do_pt,
        BpBoxes B) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float4* __restrict__ vlo = B.vlo;
    const float4* __restrict__ vhi = B.vhi;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const bool todo = B.paired[b] && !B.clok[b];
        __syncthreads();           // read by all before thread 0 sets the flag
        if (!todo) continue;
        const int v0 = vbeg[b], v1 = vbeg[b + 1], vc = cl_first(vbeg, b);
        const int e0 = ebeg[b], e1 = ebeg[b + 1], ec = cl_first(ebeg, b);
        const int t0 = tbeg[b], t1 = tbeg[b + 1], tc = cl_first(tbeg, b);
        const int nv = do_pt ? cl_count(vbeg, b) : 0, ne = do_ee ? cl_count(ebeg, b) : 0, nt = do_pt ? cl_count(tbeg, b) : 0;
        for (int j = warp; j < nv + ne + nt; j += BOX_THREADS / 32) {
            float4 l, h;
            empty_box(l, h);
            if (j < ne) {
                const int e = e0 + j * BP_CL + lane;
                if (e < e1) {
                    const int2 ed = edges[e];
                    l = fmin4(vlo[ed.x], vlo[ed.y]); h = fmax4(vhi[ed.x], vhi[ed.y]);
                }
                warp_union(l, h);
                if (lane == 0) { B.cl[1][ec + j] = l; B.ch[1][ec + j] = h; }
            } else if (j < ne + nt) {
                const int t = t0 + (j - ne) * BP_CL + lane;
                if (t < t1) {
                    const int a0 = tris[3*t], a1 = tris[3*t+1], a2 = tris[3*t+2];
                    l = fmin4(vlo[a0], fmin4(vlo[a1], vlo[a2])); h = fmax4(vhi[a0], fmax4(vhi[a1], vhi[a2]));
                }
                warp_union(l, h);
                if (lane == 0) { B.cl[2][tc + j - ne] = l; B.ch[2][tc + j - ne] = h; }
            } else {
                const int v = v0 + (j - ne - nt) * BP_CL + lane;
                if (v < v1) { l = vlo[v]; h = vhi[v]; }
                warp_union(l, h);
                if (lane == 0) { B.cl[0][vc + j - ne - nt] = l; B.ch[0][vc + j - ne - nt] = h; }
            }
        }
        if (threadIdx.x == 0) B.clok[b] = 1;
    }
}

// ---- step 3: overlapping cluster pairs of each body pair, as primitive
// ranges {first of a, first of b, counts | kind | same body}.  The counter
// is 64-bit and exact: the host grows the list once and runs the kernel
// again.  `q0`, `q1`: the slice of body pairs to expand; `c0`, `c1`: of the
// clusters of their first sides (whole groups of 32).
DV int4 cl_item(int a0, int na, int b0, int nb, int kind, int same) {
    return make_int4(a0, b0, min(na, BP_CL) | (min(nb, BP_CL) << 8) | (kind << 16) | (same << 17), 0);
}
__global__ void k_bp_clusters(const int2* __restrict__ bpairs, const int* __restrict__ npairs, int bp_cap, int q0, int q1,
                              int c0, int c1, const int* __restrict__ vbeg, const int* __restrict__ ebeg, const int* __restrict__ tbeg,
                              BpBoxes B, int do_ee, int do_pt, int4* out, long long cap, unsigned long long* count) {
    const int lane = threadIdx.x & 31;
    const int n = min(min(*npairs, bp_cap), q1);     // an overflowing pair list is rebuilt larger by the host
    // pass 0: edges of a x edges of b; 1: vertices of a x triangles of b; 2: the reverse.
    // One warp per pair and pass: three times the warps, a third of the dependent loads each.
    const int first = do_ee ? 0 : 1, np = (do_pt ? 3 : 1) - first;
    if (np <= 0) return;
    for (long long w = (long long)q0 * np + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w < (long long)n * np;
         w += (gridDim.x * blockDim.x) >> 5) {
        const int2 bp = bpairs[w / np];
        const int same = bp.x == bp.y;
        const float4 rlo = fmax4(B.blo[bp.x], B.blo[bp.y]), rhi = fmin4(B.bhi[bp.x], B.bhi[bp.y]);
        {
            const int pass = first + (int)(w % np);
            if (same && pass == 2) continue;
            const int kind = pass == 0 ? ABD_CONTACT_EE : ABD_CONTACT_PT;
            const int ba = pass == 2 ? bp.y : bp.x, bb = pass == 2 ? bp.x : bp.y;
            const int* abeg = pass == 0 ? ebeg : vbeg;
            const int* bbeg = pass == 0 ? ebeg : tbeg;
            const float4* AL = pass == 0 ? B.cl[1] : B.cl[0];
            const float4* AH = pass == 0 ? B.ch[1] : B.ch[0];
            const float4* BL = pass == 0 ? B.cl[1] : B.cl[2];
            const float4* BH = pass == 0 ? B.ch[1] : B.ch[2];
            const int na = cl_count(abeg, ba), nb = cl_count(bbeg, bb);
            const int ca = cl_first(abeg, ba), cb = cl_first(bbeg, bb);
            for (int a0 = c0; a0 < min(na, c1); a0 += 32) {
                float4 al, ah;
                empty_box(al, ah);
                if (a0 + lane < na) { al = AL[ca + a0 + lane]; ah = AH[ca + a0 + lane]; }
                const unsigned am = __ballot_sync(0xffffffffu, a0 + lane < na && overlap(al, ah, rlo, rhi));
                if (!am) continue;
                for (int b0 = 0; b0 < nb; b0 += 32) {
                    float4 bl, bh;
                    empty_box(bl, bh);
                    bool bin = b0 + lane < nb;
                    if (bin) { bl = BL[cb + b0 + lane]; bh = BH[cb + b0 + lane]; }
                    bin = bin && overlap(bl, bh, rlo, rhi);
                    if (!__any_sync(0xffffffffu, bin)) continue;
                    for (unsigned m = am; m; m &= m - 1) {
                        const int i = __ffs(m) - 1;
                        const float4 l = make_float4(__shfl_sync(0xffffffffu, al.x, i), __shfl_sync(0xffffffffu, al.y, i), __shfl_sync(0xffffffffu, al.z, i), 0.f);
                        const float4 h = make_float4(__shfl_sync(0xffffffffu, ah.x, i), __shfl_sync(0xffffffffu, ah.y, i), __shfl_sync(0xffffffffu, ah.z, i), 0.f);
                        const bool hit = bin && overlap(l, h, bl, bh) && !(same && pass == 0 && b0 + lane < a0 + i);
                        const unsigned hm = __ballot_sync(0xffffffffu, hit);
                        if (!hm) continue;
                        unsigned long long at = 0;
                        if (lane == 0) at = atomicAdd(count, (unsigned long long)__popc(hm));
                        at = __shfl_sync(0xffffffffu, at, 0) + __popc(hm & ((1u << lane) - 1));
                        if (hit && at < (unsigned long long)cap) {
                            const int pa = abeg[ba] + (a0 + i) * BP_CL, pb = bbeg[bb] + (b0 + lane) * BP_CL;
                            out[at] = cl_item(pa, abeg[ba + 1] - pa, pb, bbeg[bb + 1] - pb, kind, same);
                        }
                    }
                }
            }
        }
    }
}

// ---- step 4: one warp per cluster pair
constexpr int PRIM_THREADS = 128;
__global__ void __launch_bounds__(PRIM_THREADS) k_bp_prims(const int4* __restrict__ items,
                                                           const unsigned long long* __restrict__ nitems, long long cap, BpArgs A) {
    __shared__ int2 queue[PRIM_THREADS / 32][64];
    const int lane = threadIdx.x & 31;
    int2* Q = queue[threadIdx.x >> 5];
    const Geo& G = A.G;
    int qn = 0;                                   // queued box overlaps of this warp
    auto test = [&](int at) {
        const int2 e = Q[at];
        const int a = e.x & 0x7fffffff, b = e.y;
        if (e.x >= 0) { if (bp_ee_ok(A, min(a, b), max(a, b))) bp_emit(A, ABD_CONTACT_EE, min(a, b), max(a, b)); }
        else if (bp_pt_ok(A, a, b)) bp_emit(A, ABD_CONTACT_PT, a, b);
    };
    const long long n = min((long long)*nitems, cap);
    for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; w < n; w += ((long long)gridDim.x * blockDim.x) >> 5) {
        const int4 it = items[w];
        const int na = it.z & 0xff, nb = (it.z >> 8) & 0xff, pt = (it.z >> 16) & 1, same = (it.z >> 17) & 1;
        float4 al, ah, bl, bh;
        empty_box(al, ah);
        empty_box(bl, bh);
        if (lane < na) {
            if (pt) { al = A.vlo[it.x + lane]; ah = A.vhi[it.x + lane]; }
            else {
                const int2 ed = G.edges[it.x + lane];
                al = fmin4(__ldg(A.vlo + ed.x), __ldg(A.vlo + ed.y)); ah = fmax4(__ldg(A.vhi + ed.x), __ldg(A.vhi + ed.y));
            }
        }
        if (lane < nb) {
            if (pt) {
                const int* t = G.tris + 3L * (it.y + lane);
                const int v0 = t[0], v1 = t[1], v2 = t[2];
                bl = fmin4(__ldg(A.vlo + v0), fmin4(__ldg(A.vlo + v1), __ldg(A.vlo + v2)));
                bh = fmax4(__ldg(A.vhi + v0), fmax4(__ldg(A.vhi + v1), __ldg(A.vhi + v2)));
            } else {
                const int2 ed = G.edges[it.y + lane];
                bl = fmin4(__ldg(A.vlo + ed.x), __ldg(A.vlo + ed.y)); bh = fmax4(__ldg(A.vhi + ed.x), __ldg(A.vhi + ed.y));
            }
        }
        float4 ul = bl, uh = bh;
        warp_union(ul, uh);
        for (unsigned m = __ballot_sync(0xffffffffu, lane < na && overlap(al, ah, ul, uh)); m; m &= m - 1) {
            const int i = __ffs(m) - 1;
            const float4 l = make_float4(__shfl_sync(0xffffffffu, al.x, i), __shfl_sync(0xffffffffu, al.y, i), __shfl_sync(0xffffffffu, al.z, i), 0.f);
            const float4 h = make_float4(__shfl_sync(0xffffffffu, ah.x, i), __shfl_sync(0xffffffffu, ah.y, i), __shfl_sync(0xffffffffu, ah.z, i), 0.f);
            const bool hit = lane < nb && overlap(l, h, bl, bh) && !(same && !pt && it.x + i >= it.y + lane);
            const unsigned hm = __ballot_sync(0xffffffffu, hit);
            if (!hm) continue;
            if (hit) Q[qn + __popc(hm & ((1u << lane) - 1))] = make_int2((it.x + i) | (pt ? 0x80000000 : 0), it.y + lane);
            qn += __popc(hm);
            __syncwarp();
            if (qn >= 32) {
                test(lane);
                __syncwarp();
                qn -= 32;
                int2 rest;
                if (lane < qn) rest = Q[32 + lane];
                __syncwarp();
                if (lane < qn) Q[lane] = rest;
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (lane < qn) test(lane);
}

// ---- step 5 for lists of at most RANK_MAX hits: a key's place is the number
// of smaller keys (keys are distinct), counted by BR_SPLIT threads per key
// over the whole list and written decoded, one launch instead of a radix
// sort's histogram, scan and eight passes plus the decoding.  Counting is
// quadratic; against the sort and the decoding it takes 7 us to 22 for 256 hits,
// 15 to 102 for 4,096, 86 to 102 for 16,384 and 177 to 103 for 24,576.
constexpr int RANK_MAX = 16384, BR_THREADS = 256, BR_SPLIT = 8, BR_KEYS = BR_THREADS / BR_SPLIT;
__global__ void __launch_bounds__(BR_THREADS) k_bp_rank(int n, const unsigned long long* __restrict__ keys, int4* out, int* n_ee) {
    __shared__ unsigned long long tile[BR_THREADS * 4];
    const int k = blockIdx.x * BR_KEYS + threadIdx.x / BR_SPLIT, part = threadIdx.x % BR_SPLIT;
    const unsigned long long key = k < n ? keys[k] : 0;
    int rank = 0;
    for (int t0 = 0; t0 < n; t0 += BR_THREADS * 4) {
        const int m = min(BR_THREADS * 4, n - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += BR_THREADS) tile[i] = keys[t0 + i];
        __syncthreads();
#pragma unroll 4
        for (int i = part; i < m; i += BR_SPLIT) rank += tile[i] < key;
    }
#pragma unroll
    for (int o = BR_SPLIT / 2; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (part == 0 && k < n) {
        const int kind = (int)(key >> 62);
        out[rank] = make_int4(kind, (int)((key >> 31) & 0x7fffffffull), (int)(key & 0x7fffffffull), 0);
        // the last edge-edge pair gives their count
        if (kind == ABD_CONTACT_EE) atomicMax(n_ee, rank + 1);
    }
}

// 4. decode sorted keys into (kind, a, b) entries; count the EE prefix
__global__ void k_bp_decode(int n, const unsigned long long* __restrict__ keys, int4* out, int* n_ee) {
    GS_LOOP(i, n) {
        unsigned long long k = keys[i];
        int kind = (int)(k >> 62), a = (int)((k >> 31) & 0x7fffffffull), b = (int)(k & 0x7fffffffull);
        out[i] = make_int4(kind, a, b, 0);
        bool ee = kind == ABD_CONTACT_EE;
        bool next_ee = i + 1 < n && (int)(keys[i+1] >> 62) == ABD_CONTACT_EE;
        if (ee && !next_ee) *n_ee = (int)i + 1;
    }
}

struct BpScratch {
    void* slab = nullptr;                   // boxes, flags and counters
    BpBoxes B = {};
    int2* bpairs = nullptr; int bp_cap = 0;
    int4* items = nullptr; long long item_cap = 0;   // cluster pairs
    unsigned long long* keys = nullptr; unsigned long long* keys_s = nullptr; int key_cap = 0;
    int* cnt = nullptr;                     // [0] body pairs, [1] hits, [2] n_ee, [4..5] cluster pairs (64-bit)
    bool swept = false;                     // the boxes are those of a swept build (k_bp_boxes keeps bodies that stay put)
    void* tmp = nullptr; size_t tmp_bytes = 0;
};
constexpr long long BP_ITEM_LIMIT = 1LL << 27;     // cluster pairs held at once (2 GiB)
static BpScratch* bps(Engine* E) { return reinterpret_cast<BpScratch*>(E->bp_state); }

void eng_step_boxes(Engine* E, const float4** lo, const float4** hi) {
    BpScratch* S = bps(E);
    *lo = S && S->swept ? S->B.blo : nullptr;
    *hi = S && S->swept ? S->B.bhi : nullptr;
}

void eng_bp_free(Engine* E) {
    BpScratch* S = bps(E);
    if (!S) return;
    void* ps[] = {S->slab, S->bpairs, S->items, S->keys, S->tmp};
    for (void* p : ps) if (p) cudaFree(p);
    delete S;
    E->bp_state = nullptr;
}

static int bp_reserve(Engine* E, int bp_need, long long item_need, int key_need) {
    BpScratch* S = bps(E);
    if (!S) {
        S = new BpScratch();
        // one allocation for all boxes, flags and counters of the handle
        const size_t nb = E->nb, nv = E->nv;
        const size_t nc[3] = {nv / 32 + nb + 1, (size_t)E->ne / 32 + nb + 1, (size_t)E->nt / 32 + nb + 1};
        const size_t boxes = 2 * (nb + nv + nc[0] + nc[1] + nc[2]);
        if (cudaMalloc(&S->slab, sizeof(float4) * boxes + sizeof(int) * (8 + 3 * nb)) != cudaSuccess) {
            delete S;
            return E->fail(ABD_ERR_CUDA, "cudaMalloc body boxes");
        }
        E->bp_state = S;
        float4* at = reinterpret_cast<float4*>(S->slab);
        auto take = [&](float4*& lo, float4*& hi, size_t n) { lo = at; hi = at + n; at += 2 * n; };
        take(S->B.blo, S->B.bhi, nb);
        take(S->B.vlo, S->B.vhi, nv);
        for (int k = 0; k < 3; k++) take(S->B.cl[k], S->B.ch[k], nc[k]);
        S->cnt = reinterpret_cast<int*>(at);
        S->B.still = S->cnt + 8; S->B.paired = S->B.still + nb; S->B.clok = S->B.paired + nb;
    }
    // buffers in use by queued work are freed only after the stream drains
    if (bp_need > S->bp_cap || item_need > S->item_cap || key_need > S->key_cap) eng_stream_sync(E);
    // half as much again; a list that does not fit is an overflow, which the
    // swept list answers with a shorter step
    auto more = [](long long need, long long extra, long long limit) { return std::min(need + need / 2 + extra, limit); };
    if (bp_need > S->bp_cap) {
        const int cap = (int)more(bp_need, 1024, LIST_MAX);
        if (bp_need > cap) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "body pairs beyond the largest list");
        Replacement R;
        R.add(S->bpairs, cap);
        if (!R.commit()) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "body pairs do not fit in device memory");
        S->bp_cap = cap;
    }
    if (item_need > S->item_cap) {
        const long long cap = more(item_need, 4096, BP_ITEM_LIMIT);
        Replacement R;
        R.add(S->items, cap);
        if (!R.commit()) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "cluster pairs do not fit in device memory");
        S->item_cap = cap;
    }
    if (key_need > S->key_cap) {
        const int cap = (int)more(key_need, 4096, LIST_MAX);
        if (key_need > cap) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "pairs beyond the largest list");
        size_t tmp_bytes = 0;
        cub::DeviceRadixSort::SortKeys(nullptr, tmp_bytes, S->keys, S->keys_s, cap);
        Replacement R;
        R.add(S->keys, 2 * (size_t)cap);
        R.add_bytes(&S->tmp, tmp_bytes);
        if (!R.commit()) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "pair keys do not fit in device memory");
        S->key_cap = cap;
        S->keys_s = S->keys + cap;
        S->tmp_bytes = tmp_bytes;
    }
    return ABD_OK;
}

// the counts to pinned host memory (a copy costs 6 us with its gap, this 3)
__global__ void k_bp_send(const int* __restrict__ cnt, int* host) { if (threadIdx.x < 8) host[threadIdx.x] = cnt[threadIdx.x]; }

// Build a sorted (kind, a, b) list of EE and PT candidates into `out`
// (capacity *cap, grown through `grow`).  disp.dq null: static positions.
// mode 0: swept list with limit lim; mode 1: detection with distance filt.
// The list length comes back to the host; its EE count stays on the device
// (BpScratch::cnt[2] until the next build).
// Steps of the resting 16 x 16 net, one handle: 13.51 -> 11.85 ms per step, of
// eight nets in one handle 24.5 -> 18.1 ms, against one block per body pair
// with both bodies' primitives staged in shared memory (90 and 464 us per
// build there; boxes, pairs, clusters and primitive tests 45 and 190 us here)
// and a radix sort over 64 bits for every list (35 us for short ones, k_bp_rank
// 12 us; the sort stays for longer lists, where counting is quadratic).
static int bp_build(Engine* E, const BpDisp& disp, double lim, double filt, int mode, int4*& out, int& cap, int& n_out,
                    int (*grow)(Engine*, int)) {
    cudaStream_t s = E->stream;
    const AbdParams& P = E->P;
    int rc;
    if ((rc = bp_reserve(E, 4 * E->nb + 1024, 64LL * E->nb + 4096, std::max(cap, 4096)))) return rc;
    BpScratch* S = bps(E);
    const float pad = (float)(0.5 * lim);
    const int do_ee = P.contact_ee && E->ne > 0, do_pt = P.contact_pt && E->nt > 0;
    // the positions are those the last swept build's step led to, so a body
    // that stays put in both has the same boxes
    const int keep = mode == 0 && S->swept && E->sw_valid;
    S->swept = false;
    const int body_grid = std::min(E->nb, NUM_SMS * 16);
    k_bp_boxes<<<body_grid, BOX_THREADS, 0, s>>>(E->nb, E->bd_vbeg, E->x, disp, pad, keep, S->B, S->cnt);
    E->launches++;
    for (int attempt = 0; attempt < 8; attempt++) {
        if (attempt > 0) CUDA_TRY(cudaMemsetAsync(S->cnt, 0, sizeof(int) * 8, s));
        k_body_pairs<<<grid_for(32L * E->nb), 256, 0, s>>>(E->nb, E->bscene, E->sc_body_begin, S->B.blo, S->B.bhi,
                                                            P.self_contact, S->bpairs, S->bp_cap, S->cnt, S->B.paired);
        k_bp_clboxes<<<body_grid, BOX_THREADS, 0, s>>>(E->nb, E->bd_vbeg, E->bd_ebeg, E->bd_tbeg, E->edges, E->tris, do_ee,
                                                       do_pt, S->B);
        BpArgs A;
        A.G = eng_geo(E); A.pmag = E->pmag; A.vlo = S->B.vlo; A.vhi = S->B.vhi;
        A.lim = lim; A.filt = filt; A.mode = mode; A.f32 = P.ee_f32;
        A.out = S->keys; A.cap = S->key_cap; A.count = S->cnt + 1;
        unsigned long long* nitems = reinterpret_cast<unsigned long long*>(S->cnt + 4);
        auto expand = [&](int q0, int q1, int c0, int c1) {
            k_bp_clusters<<<NUM_SMS * 4, 256, 0, s>>>(S->bpairs, S->cnt, S->bp_cap, q0, q1, c0, c1, E->bd_vbeg, E->bd_ebeg, E->bd_tbeg,
                                                       S->B, do_ee, do_pt, S->items, S->item_cap, nitems);
            k_bp_prims<<<NUM_SMS * 8, PRIM_THREADS, 0, s>>>(S->items, nitems, S->item_cap, A);
            E->launches += 2;
        };
        expand(0, INT_MAX, 0, INT_MAX);
        k_bp_send<<<1, 32, 0, s>>>(S->cnt, E->hcnt->bp);
        E->launches += 3;
        CUDA_TRY(eng_stream_sync(E));
        const int npairs = E->hcnt->bp[0];
        long long items;
        memcpy(&items, E->hcnt->bp + 4, sizeof items);
        if (npairs > S->bp_cap || (items > S->item_cap && S->item_cap < BP_ITEM_LIMIT) || E->hcnt->bp[1] > S->key_cap) {
            if ((rc = bp_reserve(E, npairs, std::min(items, BP_ITEM_LIMIT), E->hcnt->bp[1]))) return rc;
            continue;
        }
        if (items > S->item_cap) {
            // more cluster pairs than the list may hold: slices of body pairs
            // small enough to fit whatever they overlap, and of a pair's
            // clusters where a single one would not (one cluster meets at most
            // `row` others, so a group of 32 fits up to 130 million primitives)
            auto most = [&](int n) { return (long long)n / 32 + 1; };
            const long long row = most(E->ne) + 2 * most(E->nt), rows = std::max(most(E->ne), most(E->nv)), per = row * rows;
            const int step = (int)std::max<long long>(1, S->item_cap / per);
            const long long cstep = per <= S->item_cap ? rows + 32 : std::max<long long>(32, S->item_cap / row / 32 * 32);
            CUDA_TRY(cudaMemsetAsync(S->cnt + 1, 0, sizeof(int), s));
            for (int q0 = 0; q0 < npairs; q0 += step)
                for (long long c0 = 0; c0 < rows; c0 += cstep) {
                    CUDA_TRY(cudaMemsetAsync(nitems, 0, sizeof(long long), s));
                    expand(q0, std::min(npairs, q0 + step), (int)c0, (int)std::min<long long>(c0 + cstep, INT_MAX));
                    k_bp_send<<<1, 32, 0, s>>>(S->cnt, E->hcnt->bp);
                    E->launches++;
                    CUDA_TRY(eng_stream_sync(E));
                    memcpy(&items, E->hcnt->bp + 4, sizeof items);
                    if (items > S->item_cap) return E->fail(ABD_ERR_CONTACT_OVERFLOW, "body-pair broad phase: one body pair's cluster pairs do not fit");
                }
            if (E->hcnt->bp[1] > S->key_cap) {
                if ((rc = bp_reserve(E, npairs, 0, E->hcnt->bp[1]))) return rc;
                continue;
            }
        }
        const int n = E->hcnt->bp[1];
        if (n > cap) { if ((rc = grow(E, n))) return rc; }
        if (n > 0 && n <= RANK_MAX) {
            k_bp_rank<<<(n + BR_KEYS - 1) / BR_KEYS, BR_THREADS, 0, s>>>(n, S->keys, out, S->cnt + 2);
            E->launches++;
        } else if (n > 0) {
            size_t bytes = S->tmp_bytes;
            CUDA_TRY(cub::DeviceRadixSort::SortKeys(S->tmp, bytes, S->keys, S->keys_s, n, 0, 64, s));
            k_bp_decode<<<grid_for(n), 256, 0, s>>>(n, S->keys_s, out, S->cnt + 2);
            E->launches += 2;
        }
        n_out = n;
        S->swept = mode == 0;
        return ABD_OK;
    }
    return E->fail(ABD_ERR_CONTACT_OVERFLOW, "body-pair broad phase did not fit after growing");
}

static int grow_sw(Engine* E, int need) { return eng_grow_swept(E, need); }
static int grow_ct(Engine* E, int need) { return eng_grow_contacts(E, need); }

// swept list along the displacement sign * J dq (left in E->pv), limit lim;
// bodies of scenes flagged done do not move
int eng_swept_bp(Engine* E, const double* dq, double sign, const int* done, double lim) {
    int n = 0;
    const BpDisp disp = {dq, sign, E->xbar, E->mass, E->bscene, done, E->pv, E->pmag};
    int rc = bp_build(E, disp, lim, lim, 0, E->sw, E->sw_cap, n, grow_sw);
    if (rc) return rc;
    E->n_sw = n; E->sw_valid = true;
    return ABD_OK;
}

__global__ void k_bp_counts(Counters* cnt, const int* __restrict__ n_ee_dev, int n) {
    if (threadIdx.x == 0 && blockIdx.x == 0) { int n_ee = *n_ee_dev; cnt->n_ee = n_ee; cnt->n_pt = n - n_ee; cnt->overflow = 0; }
}

// full detection at the current positions with filter filt
int eng_detect_bp(Engine* E, double filt) {
    int rc = eng_transform(E);
    if (rc) return rc;
    CUDA_TRY(cudaMemsetAsync(E->dcnt, 0, DETECT_COUNTER_BYTES, E->stream));
    double lim = filt * (1.0 + 1e-6) + 1e-7;
    int n = 0;
    if ((rc = bp_build(E, BpDisp{}, lim, filt, 1, E->contacts, E->cap, n, grow_ct))) return rc;
    k_bp_counts<<<1, 32, 0, E->stream>>>(E->dcnt, bps(E)->cnt + 2, n);
    E->launches++;
    return eng_pg_candidates(E, filt);
}

// ------------------------------------------------------------------ contact groups of the line search
//
// Two bodies belong to one group when their boxes swept over the listed
// step x .. x + p, padded by half the candidate distance on every side,
// overlap (transitively).  Bodies of different groups stay more than the
// candidate distance apart for any pair of step fractions in [0, 1], so no
// listed pair, barrier term or CCD bound couples them and each group can
// take its own step length.  The union-find hooks the larger root under the
// smaller with atomicCAS, so a group's root is its smallest body index.

DV int grp_find(const int* parent, int x, int limit) {
    for (int k = 0; k < limit; k++) {
        int p = __ldcg(parent + x);
        if (p == x) return x;
        x = p;
    }
    return x;
}

__global__ void k_grp_init(int nb, int* parent) { GS_LOOP(b, nb) parent[b] = (int)b; }

// one warp per body a: every later body b of the scene whose box overlaps
__global__ void k_grp_union(int nb, const int* __restrict__ bscene, const int* __restrict__ sc_body_begin,
                            const float4* __restrict__ blo, const float4* __restrict__ bhi, int* parent, Counters* cnt) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    for (int a = warp; a < nb; a += (gridDim.x * blockDim.x) >> 5) {
        int end = sc_body_begin[bscene[a] + 1];
        float4 al = blo[a], ah = bhi[a];
        for (int b = a + 1 + lane; b < end; b += 32) {
            if (!overlap(al, ah, blo[b], bhi[b])) continue;
            // every failed CAS means a root was hooked, which happens at
            // most nb - 1 times in total
            int ra = a, rb = b;
            bool ok = false;
            for (int k = 0; k <= nb; k++) {
                ra = grp_find(parent, ra, nb + 1); rb = grp_find(parent, rb, nb + 1);
                if (ra == rb) { ok = true; break; }
                if (ra < rb) { int t = ra; ra = rb; rb = t; }
                int old = atomicCAS(parent + ra, ra, rb);
                if (old == ra) { ok = true; break; }
                ra = old;
            }
            if (!ok) atomicExch(&cnt->grp_fail, 1);
        }
    }
}

// root per body; a unit (a root body) joins the line search when its scene
// is still iterating, every other slot is skipped
__global__ void k_grp_finish(int nb, int* parent, const int* __restrict__ bscene, const int* __restrict__ done,
                             int* udone) {
    GS_LOOP(b, nb) {
        int r = grp_find(parent, (int)b, nb + 1);
        parent[b] = r;
        udone[b] = (r != (int)b) || done[bscene[b]];
    }
}

void eng_groups_free(Engine* E) {
    void* ps[] = {E->grp, E->gscd, E->gsci, E->grp_lo, E->grp_hi};
    for (void* p : ps) if (p) cudaFree(p);
    E->grp = nullptr; E->gscd = nullptr; E->gsci = nullptr; E->grp_lo = nullptr; E->grp_hi = nullptr;
}

// groups of the step listed by the last eng_swept (positions E->x, step
// E->pv); needs contiguous per-body vertex ranges
int eng_groups(Engine* E, const int* done) {
    if (!E->bd_ok) return E->fail(ABD_ERR_INVALID_ARG, "ls_groups needs contiguous per-body vertex ranges");
    int nb = E->nb;
    cudaStream_t s = E->stream;
    if (!E->grp) {
        if (cudaMalloc(&E->grp, sizeof(int) * nb) != cudaSuccess ||
            cudaMalloc(&E->gscd, sizeof(double) * SD_COUNT * nb) != cudaSuccess ||
            cudaMalloc(&E->gsci, sizeof(int) * SI_COUNT * nb) != cudaSuccess ||
            cudaMalloc(&E->grp_lo, sizeof(float4) * nb) != cudaSuccess ||
            cudaMalloc(&E->grp_hi, sizeof(float4) * nb) != cudaSuccess) {
            eng_groups_free(E);
            return E->fail(ABD_ERR_CUDA, "cudaMalloc contact groups");
        }
        CUDA_TRY(cudaMemsetAsync(E->gscd, 0, sizeof(double) * SD_COUNT * nb, s));
        CUDA_TRY(cudaMemsetAsync(E->gsci, 0, sizeof(int) * SI_COUNT * nb, s));
    }
    double lim = E->P.cand_dist * (1.0 + 1e-6) + 1e-7;
    float pad = (float)(0.5 * lim);
    k_grp_init<<<grid_for(nb), 256, 0, s>>>(nb, E->grp);
    k_body_boxes<<<grid_for(32L * nb), 256, 0, s>>>(nb, E->bd_vbeg, E->x, E->pv, pad, E->grp_lo, E->grp_hi);
    k_grp_union<<<grid_for(32L * nb), 256, 0, s>>>(nb, E->bscene, E->sc_body_begin, E->grp_lo, E->grp_hi, E->grp, E->dcnt);
    k_grp_finish<<<grid_for(nb), 256, 0, s>>>(nb, E->grp, E->bscene, done, E->gsci + SI_DONE * nb);
    E->launches += 4;
    return ABD_OK;
}
