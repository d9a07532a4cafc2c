// detect.cu — vertex transform, uniform-grid broad phase, candidate pairs,
// contact energy, the ordered filter of listed candidates and the intersection check.
//
//  transform ............ abd_simple.py:26-35
//  EE candidates ........ contact.py:25-32, :143-169 (float32 predicate, i<j,
//                         no shared vertex, distance < (thickness+buffer)*2)
//  PT / half-space ...... no reference counterpart
//  contact energy ....... abd.py:66-75
//
// The reference refits a Warp LBVH and appends pairs with an atomic counter
// (unordered, capacity 10000 with wrap-around).  Here every detection
// rebuilds a hashed uniform grid (one radix sort), counts pairs per query
// item, scans, and writes each item's pairs in index order, so the list is
// sorted and exact-size; overflow is reported instead of wrapping.
#include "energy.cuh"
#include <cub/cub.cuh>

// ------------------------------------------------------------------ transform
__global__ void k_transform(int nv, const double* __restrict__ xbar, const int* __restrict__ vbody,
                            const double* __restrict__ st, double* __restrict__ x, float4* __restrict__ xf) {
    GS_LOOP(v, nv) {
        const double* s = st + (long)ST_STRIDE * vbody[v] + ST_NXT;
        double xb0 = xbar[3*v], xb1 = xbar[3*v+1], xb2 = xbar[3*v+2];
        double o[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            double t = s[ST_C + k];
            t = __fma_rn(s[ST_Q + 0 + k], xb0, t);
            t = __fma_rn(s[ST_Q + 3 + k], xb1, t);
            t = __fma_rn(s[ST_Q + 6 + k], xb2, t);
            o[k] = t;
        }
        x[3*v] = o[0]; x[3*v+1] = o[1]; x[3*v+2] = o[2];
        xf[v] = make_float4(__double2float_rn(o[0]), __double2float_rn(o[1]), __double2float_rn(o[2]), 0.f);
    }
}

int eng_body_energy(Engine* E, double* Eo, const int* skip);
int eng_pg_energy(Engine* E, double* Eo, const int* skip);
int eng_pg_candidates(Engine* E, double filt);

// Vertex positions of the nxt state.  The line search leaves them behind with
// every state it writes, so they are formed here only after the state came
// from outside.
int eng_transform(Engine* E) {
    if (E->x_fresh) return ABD_OK;
    k_transform<<<grid_for(E->nv), 256, 0, E->stream>>>(E->nv, E->xbar, E->vbody, E->st, E->x, E->xf);
    E->launches++;
    E->x_fresh = true;
    return ABD_OK;
}

// ------------------------------------------------------------------ boxes
DV float f_rd(double v) { return __double2float_rd(v); }
DV float f_ru(double v) { return __double2float_ru(v); }

// Edge boxes, both stored and queried.  f32 mode boxes the float copies
// exactly; f64 mode rounds outward.  pad is added on every side.
__global__ void k_edge_boxes(int ne, const int2* __restrict__ edges, const double* __restrict__ x,
                             const float4* __restrict__ xf, const int* __restrict__ escene, float pad, int f32,
                             float4* lo, float4* hi, int* scene, float* cell) {
    float ext = 0.f;
    GS_LOOP(e, ne) {
        int2 ed = edges[e];
        float l[3], h[3];
        if (f32) {
            float4 a = xf[ed.x], b = xf[ed.y];
            l[0] = fminf(a.x, b.x); l[1] = fminf(a.y, b.y); l[2] = fminf(a.z, b.z);
            h[0] = fmaxf(a.x, b.x); h[1] = fmaxf(a.y, b.y); h[2] = fmaxf(a.z, b.z);
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                double a = x[3*ed.x+k], b = x[3*ed.y+k];
                l[k] = f_rd(fmin(a, b)); h[k] = f_ru(fmax(a, b));
            }
        }
        float4 L = make_float4(__fsub_rd(l[0], pad), __fsub_rd(l[1], pad), __fsub_rd(l[2], pad), 0.f);
        float4 Hh = make_float4(__fadd_ru(h[0], pad), __fadd_ru(h[1], pad), __fadd_ru(h[2], pad), 0.f);
        lo[e] = L; hi[e] = Hh; scene[e] = escene[e];
        ext = fmaxf(ext, fmaxf(Hh.x - L.x, fmaxf(Hh.y - L.y, Hh.z - L.z)));
    }
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if ((threadIdx.x & 31) == 0 && ext > 0.f) atomic_max_pos(cell, ext);
}

__global__ void k_tri_boxes(int nt, const int* __restrict__ tris, const double* __restrict__ x,
                            const int* __restrict__ tscene, float pad, float4* lo, float4* hi, int* scene, float* cell) {
    float ext = 0.f;
    GS_LOOP(t, nt) {
        int a = tris[3*t], b = tris[3*t+1], c = tris[3*t+2];
        float l[3], h[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            double va = x[3*a+k], vb = x[3*b+k], vc = x[3*c+k];
            l[k] = __fsub_rd(f_rd(fmin(va, fmin(vb, vc))), pad);
            h[k] = __fadd_ru(f_ru(fmax(va, fmax(vb, vc))), pad);
        }
        lo[t] = make_float4(l[0], l[1], l[2], 0.f); hi[t] = make_float4(h[0], h[1], h[2], 0.f); scene[t] = tscene[t];
        ext = fmaxf(ext, fmaxf(h[0] - l[0], fmaxf(h[1] - l[1], h[2] - l[2])));
    }
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if ((threadIdx.x & 31) == 0 && ext > 0.f) atomic_max_pos(cell, ext);
}

__global__ void k_point_boxes(int nv, const double* __restrict__ x, const int* __restrict__ vscene, float pad,
                              float4* lo, float4* hi, int* scene, float* cell) {
    float ext = 0.f;
    GS_LOOP(v, nv) {
        float l[3], h[3];
#pragma unroll
        for (int k = 0; k < 3; k++) { l[k] = __fsub_rd(f_rd(x[3*v+k]), pad); h[k] = __fadd_ru(f_ru(x[3*v+k]), pad); }
        lo[v] = make_float4(l[0], l[1], l[2], 0.f); hi[v] = make_float4(h[0], h[1], h[2], 0.f); scene[v] = vscene[v];
        ext = fmaxf(ext, fmaxf(h[0] - l[0], fmaxf(h[1] - l[1], h[2] - l[2])));
    }
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if ((threadIdx.x & 31) == 0 && ext > 0.f) atomic_max_pos(cell, ext);
}

// ------------------------------------------------------------------ grid build
__global__ void k_grid_keys(int n, const float4* __restrict__ lo, const int* __restrict__ scene, float* cell,
                            uint32_t mask, uint32_t* keys, int* vals) {
    float h = fmaxf(*cell, 1e-6f);
    GS_LOOP(i, n) {
        float4 l = lo[i];
        uint32_t key = cell_hash(scene[i], (int)floorf(l.x / h), (int)floorf(l.y / h), (int)floorf(l.z / h)) & mask;
        keys[i] = key; vals[i] = (int)i;
    }
}
__global__ void k_cell_floor(float* cell) { if (threadIdx.x == 0 && blockIdx.x == 0) *cell = fmaxf(*cell, 1e-6f); }
__global__ void k_grid_ranges(int n, const uint32_t* __restrict__ keys, int* bstart, int* bend) {
    GS_LOOP(i, n) {
        uint32_t k = keys[i];
        if (i == 0 || keys[i-1] != k) bstart[k] = (int)i;
        if (i == n - 1 || keys[i+1] != k) bend[k] = (int)i + 1;
    }
}

int eng_grid_build(Engine* E, Grid& G) {
    if (G.n == 0) return ABD_OK;
    cudaStream_t s = E->stream;
    k_cell_floor<<<1, 32, 0, s>>>(G.cell);
    k_grid_keys<<<grid_for(G.n), 256, 0, s>>>(G.n, G.lo, G.scene, G.cell, (uint32_t)(G.H - 1), G.keys, G.vals);
    size_t bytes = E->cub_bytes;
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(E->cub_tmp, bytes, G.keys, G.keys_s, G.vals, G.vals_s, G.n, 0, G.bits, s));
    CUDA_TRY(cudaMemsetAsync(G.bstart, 0xFF, sizeof(int) * G.H, s));
    k_grid_ranges<<<grid_for(G.n), 256, 0, s>>>(G.n, G.keys_s, G.bstart, G.bend);
    E->launches += 4;
    return ABD_OK;
}
GridView eng_view(const Grid& G) {
    return GridView{G.lo, G.hi, G.scene, G.cell, G.vals_s, G.bstart, G.bend, (uint32_t)(G.H - 1)};
}

// ------------------------------------------------------------------ pair queries
// mode 0: count into qcount; mode 1: write sorted pairs at qoff + base
__global__ void k_ee_pairs(int ne, GridView GV, Geo G, const float4* __restrict__ qlo, const float4* __restrict__ qhi,
                           const int* __restrict__ qscene, int f32, int self_contact, double filt, int mode,
                           int* qcount, const int* qoff, int base_slot, const Counters* cnt, int cap,
                           int4* out, int* overflow) {
    GS_LOOP(i, ne) {
        int c = 0;
        int base = 0;
        if (mode == 1) {
            base = (base_slot == 0 ? 0 : cnt->n_ee) + qoff[i];
        }
        int ii = (int)i;
        grid_visit(GV, qlo[i], qhi[i], qscene[i], [&](int j) {
            if (j <= ii) return;
            double s, t, d;
            if (!ee_test(G, ii, j, f32, self_contact, filt, s, t, d)) return;
            if (mode == 1) {
                int at = base + c;
                if ((unsigned)at < (unsigned)cap) out[at] = make_int4(ABD_CONTACT_EE, ii, j, 0);
                else *overflow = 1;
            }
            c++;
        });
        if (mode == 0) qcount[i] = c;
        else if (c > 1) {
            // insertion sort of this item's segment by partner index
            int lo = base, hi = min(base + c, cap);
            for (int k = lo + 1; k < hi; k++) {
                int4 v = out[k]; int m = k - 1;
                while (m >= lo && out[m].z > v.z) { out[m+1] = out[m]; m--; }
                out[m+1] = v;
            }
        }
    }
}

__global__ void k_pt_pairs(int nv, GridView GV, Geo G, const float4* __restrict__ qlo, const float4* __restrict__ qhi,
                           const int* __restrict__ qscene, int self_contact, double filt, int mode,
                           int* qcount, const int* qoff, const Counters* cnt, int cap, int4* out, int* overflow) {
    GS_LOOP(p, nv) {
        int c = 0, base = 0;
        if (mode == 1) base = cnt->n_ee + qoff[p];
        int pp = (int)p;
        grid_visit(GV, qlo[p], qhi[p], qscene[p], [&](int t) {
            if (!pt_test(G, pp, t, self_contact, filt)) return;
            if (mode == 1) {
                int at = base + c;
                if ((unsigned)at < (unsigned)cap) out[at] = make_int4(ABD_CONTACT_PT, pp, t, 0);
                else *overflow = 1;
            }
            c++;
        });
        if (mode == 0) qcount[p] = c;
        else if (c > 1) {
            int lo = base, hi = min(base + c, cap);
            for (int k = lo + 1; k < hi; k++) {
                int4 v = out[k]; int m = k - 1;
                while (m >= lo && out[m].z > v.z) { out[m+1] = out[m]; m--; }
                out[m+1] = v;
            }
        }
    }
}

__global__ void k_store_count(const int* qoff, int n, int slot, Counters* cnt) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int v = qoff[n];
        if (slot == 0) cnt->n_ee = v;
        else cnt->n_pt = v;
    }
}

// ------------------------------------------------------------------ ordered filter
// The candidates that survive among the listed pairs (EE, then PT) and then
// those of the vertices near a half-space (by vertex, then plane), in order
// and in two launches.  k_filter_count tests every item: a tile of pairs per
// block, whose survivors it keeps as bits, or a tile of vertices; the block
// that finishes last turns the tiles' counts into places and sets the
// counters.  k_filter_write copies the survivors of its tile there; most
// tiles have none.  (Flags, a scan and a copy per kind with their clears took eight
// nodes of an iteration: eight cubes 31 -> 12 us with the gaps, the resting 16 x 16
// net 28 -> 13, 512 scenes of 1.6 million vertices 48 -> 30.)
constexpr int FL_THREADS = 256;
constexpr int FL_VERTS = 4 * FL_THREADS;         // vertices of a tile
struct FilterArgs {
    int n; const int4* list; int f32, self_contact;  // listed pairs; n < 0: EE and PT are counted already
    int list_tiles, vert_tiles;
    int nv; const int* vscene; double filt;
    Geo G;
    uint32_t* keep;                              // survivors of the list, a bit each
    int *list_at, *ee, *vert_at;                 // per tile: count, then place; EE survivors
    int4* out; int cap; Counters* cnt;
};
DV int pg_count(const FilterArgs& A, int v) {
    const int s = A.vscene[v], p1 = A.G.sc_plane_begin[s + 1];
    int c = 0;
    for (int pl = A.G.sc_plane_begin[s]; pl < p1; pl++) {
        const double* n = A.G.planes + 4*pl;
        const double d = n[0] * A.G.x[3*v] + n[1] * A.G.x[3*v+1] + n[2] * A.G.x[3*v+2] - n[3];
        c += d < A.filt;
    }
    return c;
}
// exclusive sum over the block's threads and the block's total; every thread calls it
DV int block_scan(int v, int* sh, int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) { int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
    __syncthreads();                             // sh is free
    if (lane == 31) sh[w] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int k = 0; k < FL_THREADS / 32; k++) { if (k < w) before += sh[k]; total += sh[k]; }
    return before + incl - v;
}
// counts at `at` (of other blocks) to places from `base` on; returns the end
DV int places(int* at, int n, int base, int* sh) {
    for (int t = 0; t < n; t += FL_THREADS) {
        const int k = t + threadIdx.x;
        int total, e = block_scan(k < n ? __ldcg(at + k) : 0, sh, total);
        if (k < n) at[k] = base + e;
        base += total;
    }
    return base;
}
__global__ void __launch_bounds__(FL_THREADS) k_filter_count(FilterArgs A) {
    __shared__ int sh[FL_THREADS / 32];
    const int tile = blockIdx.x, tid = threadIdx.x;
    if (tile < A.list_tiles) {
        const int c = tile * FL_THREADS + tid;
        bool keep = false, ee = false;
        if (c < A.n) {
            const int4 C = A.list[c];
            ee = C.x == ABD_CONTACT_EE;
            if (ee) { double s, t, d; keep = ee_test(A.G, C.y, C.z, A.f32, A.self_contact, A.filt, s, t, d); }
            else keep = pt_test(A.G, C.y, C.z, A.self_contact, A.filt);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if ((tid & 31) == 0 && c < A.n) A.keep[c >> 5] = m;
        const int kept = __syncthreads_count(keep), kept_ee = __syncthreads_count(keep && ee);
        if (tid == 0) { A.list_at[tile] = kept; A.ee[tile] = kept_ee; }
    } else if (tile < A.list_tiles + A.vert_tiles) {
        const int v0 = (tile - A.list_tiles) * FL_VERTS + tid;
        int c = 0;
#pragma unroll
        for (int j = 0; j < FL_VERTS / FL_THREADS; j++) { const int v = v0 + j * FL_THREADS; if (v < A.nv) c += pg_count(A, v); }
        int total;
        block_scan(c, sh, total);
        if (tid == 0) A.vert_at[tile - A.list_tiles] = total;
    }
    if (!last_block(&A.cnt->ticket)) return;
    int n_ee = 0, base = 0;
    if (A.n < 0) base = A.cnt->n_ee + A.cnt->n_pt;
    else {
        int e = 0;
        for (int k = tid; k < A.list_tiles; k += FL_THREADS) e += __ldcg(A.ee + k);
        block_scan(e, sh, n_ee);
        base = places(A.list_at, A.list_tiles, 0, sh);
    }
    const int end = places(A.vert_at, A.vert_tiles, base, sh);
    if (tid == 0) {
        if (A.n >= 0) { A.cnt->n_ee = n_ee; A.cnt->n_pt = base - n_ee; A.cnt->overflow = 0; }
        A.cnt->n_pg = end - base;
        A.cnt->n_total = end;
        if (end > A.cap) A.cnt->overflow = 1;
    }
}
__global__ void __launch_bounds__(FL_THREADS) k_filter_write(FilterArgs A) {
    __shared__ int sh[FL_THREADS / 32];
    const int tile = blockIdx.x, tid = threadIdx.x;
    if (tile < A.list_tiles) {
        const int c = tile * FL_THREADS + tid, w0 = tile * (FL_THREADS / 32), nw = (A.n + 31) / 32;
        const unsigned m = c < A.n ? A.keep[c >> 5] : 0;
        if (!(m >> (tid & 31) & 1)) return;
        int at = A.list_at[tile] + __popc(m & ((1u << (tid & 31)) - 1));
        for (int w = w0; w < (c >> 5) && w < nw; w++) at += __popc(A.keep[w]);
        if ((unsigned)at < (unsigned)A.cap) A.out[at] = A.list[c];
        return;
    }
    const int t = tile - A.list_tiles;
    int base = A.vert_at[t];
    const int end = t + 1 < A.vert_tiles ? A.vert_at[t + 1] : A.cnt->n_total;
    if (base == end) return;
    for (int j = 0; j < FL_VERTS / FL_THREADS; j++) {
        const int v = t * FL_VERTS + j * FL_THREADS + tid;
        int total, at = base + block_scan(v < A.nv ? pg_count(A, v) : 0, sh, total);
        base += total;
        if (v >= A.nv) continue;
        const int s = A.vscene[v], p1 = A.G.sc_plane_begin[s + 1];
        for (int pl = A.G.sc_plane_begin[s]; pl < p1; pl++) {
            const double* n = A.G.planes + 4*pl;
            const double d = n[0] * A.G.x[3*v] + n[1] * A.G.x[3*v+1] + n[2] * A.G.x[3*v+2] - n[3];
            if (!(d < A.filt)) continue;
            if ((unsigned)at < (unsigned)A.cap) A.out[at] = make_int4(ABD_CONTACT_PG, v, pl, 0);
            at++;
        }
    }
}

static Geo geo(Engine* E) {
    return Geo{E->x, E->xf, E->edges, E->tris, E->vbody, E->bscene, E->planes, E->sc_plane_begin, E->mass, E->xbar};
}

static int scan_counts(Engine* E, int* qcount, int* qoff, int n) {
    size_t bytes = E->cub_bytes;
    CUDA_TRY(cub::DeviceScan::ExclusiveSum(E->cub_tmp, bytes, qcount, qoff, n + 1, E->stream));
    E->launches++;
    return ABD_OK;
}

// Build the EE grid (edges stored and queried) at the current positions.
static int build_ee_grid(Engine* E, double filt) {
    Grid& G = E->gee;
    if (G.n == 0) return ABD_OK;
    float pad = (float)(0.5 * filt * (1.0 + 1e-6) + 1e-7);
    CUDA_TRY(cudaMemsetAsync(G.cell, 0, sizeof(float), E->stream));
    k_edge_boxes<<<grid_for(G.n), 256, 0, E->stream>>>(G.n, E->edges, E->x, E->xf, E->edge_scene, pad, E->P.ee_f32,
                                                       G.lo, G.hi, G.scene, G.cell);
    E->launches++;
    return eng_grid_build(E, G);
}
static int build_pt_grid(Engine* E, double filt) {
    Grid& G = E->gpt;
    if (G.n == 0) return ABD_OK;
    float pad = (float)(0.5 * filt * (1.0 + 1e-6) + 1e-7);
    CUDA_TRY(cudaMemsetAsync(G.cell, 0, sizeof(float), E->stream));
    k_tri_boxes<<<grid_for(G.n), 256, 0, E->stream>>>(G.n, E->tris, E->x, E->tri_scene, pad, G.lo, G.hi, G.scene, G.cell);
    k_point_boxes<<<grid_for(G.nq), 256, 0, E->stream>>>(G.nq, E->x, E->vscene, pad, G.qlo, G.qhi, G.qscene, G.cell);
    E->launches += 2;
    return eng_grid_build(E, G);
}

int eng_detect(Engine* E, double filt) {
    int rc;
    cudaStream_t s = E->stream;
    if ((rc = eng_transform(E))) return rc;
    CUDA_TRY(cudaMemsetAsync(E->dcnt, 0, DETECT_COUNTER_BYTES, s));
    Geo G = geo(E);
    int f32 = E->P.ee_f32, sc = E->P.self_contact;
    if (E->P.contact_ee && E->ne > 1) {
        if ((rc = build_ee_grid(E, filt))) return rc;
        Grid& g = E->gee;
        k_ee_pairs<<<grid_for(E->ne, 128), 128, 0, s>>>(E->ne, eng_view(g), G, g.lo, g.hi, g.scene, f32, sc, filt, 0,
                                                         g.qcount, nullptr, 0, E->dcnt, E->cap, E->contacts, &E->dcnt->overflow);
        CUDA_TRY(cudaMemsetAsync(g.qcount + E->ne, 0, sizeof(int), s));
        if ((rc = scan_counts(E, g.qcount, g.qoff, E->ne))) return rc;
        k_store_count<<<1, 32, 0, s>>>(g.qoff, E->ne, 0, E->dcnt);
        k_ee_pairs<<<grid_for(E->ne, 128), 128, 0, s>>>(E->ne, eng_view(g), G, g.lo, g.hi, g.scene, f32, sc, filt, 1,
                                                         g.qcount, g.qoff, 0, E->dcnt, E->cap, E->contacts, &E->dcnt->overflow);
        E->launches += 3;
    }
    if (E->P.contact_pt && E->nt > 0) {
        if ((rc = build_pt_grid(E, filt))) return rc;
        Grid& g = E->gpt;
        k_pt_pairs<<<grid_for(E->nv, 128), 128, 0, s>>>(E->nv, eng_view(g), G, g.qlo, g.qhi, g.qscene, sc, filt, 0,
                                                         g.qcount, nullptr, E->dcnt, E->cap, E->contacts, &E->dcnt->overflow);
        CUDA_TRY(cudaMemsetAsync(g.qcount + E->nv, 0, sizeof(int), s));
        if ((rc = scan_counts(E, g.qcount, g.qoff, E->nv))) return rc;
        k_store_count<<<1, 32, 0, s>>>(g.qoff, E->nv, 1, E->dcnt);
        k_pt_pairs<<<grid_for(E->nv, 128), 128, 0, s>>>(E->nv, eng_view(g), G, g.qlo, g.qhi, g.qscene, sc, filt, 1,
                                                         g.qcount, g.qoff, E->dcnt, E->cap, E->contacts, &E->dcnt->overflow);
        E->launches += 3;
    }
    return eng_pg_candidates(E, filt);
}

int eng_filter(Engine* E, int n_list, double filt) {
    FilterArgs A;
    A.n = n_list; A.list = E->sw; A.f32 = E->P.ee_f32; A.self_contact = E->P.self_contact;
    A.list_tiles = n_list > 0 ? (n_list + FL_THREADS - 1) / FL_THREADS : 0;
    A.vert_tiles = E->npl > 0 ? (E->nv + FL_VERTS - 1) / FL_VERTS : 0;
    A.nv = E->nv; A.vscene = E->vscene; A.filt = filt; A.G = geo(E);
    A.keep = (uint32_t*)E->sw_flag; A.list_at = E->sw_off; A.ee = E->sw_off + A.list_tiles;
    A.vert_at = E->gpt.qoff;                     // the PT query's, free here
    A.out = E->contacts; A.cap = E->cap; A.cnt = E->dcnt;
    const int tiles = A.list_tiles + A.vert_tiles;
    k_filter_count<<<std::max(tiles, 1), FL_THREADS, 0, E->stream>>>(A);
    if (tiles > 0) k_filter_write<<<tiles, FL_THREADS, 0, E->stream>>>(A);
    E->launches += 1 + (tiles > 0);
    return ABD_OK;
}

// half-space candidates appended after EE and PT, then the total
int eng_pg_candidates(Engine* E, double filt) { return eng_filter(E, -1, filt); }

// ------------------------------------------------------------------ energies
__global__ void k_body_energy(int nb, const double* __restrict__ st, const double* __restrict__ mass,
                              const double* __restrict__ J, const int* __restrict__ bscene, BodyTerms T, const int* done,
                              double* E) {
    for (long base = (long)blockIdx.x * blockDim.x; base < nb; base += (long)gridDim.x * blockDim.x) {
        long b = base + threadIdx.x;
        bool valid = b < nb;
        int s = valid ? bscene[b] : 0;
        double e = 0, en = 0;
        if (valid && !done[s]) body_energy(st + ST_STRIDE * b, mass[b], J[b], T, e, en);
        else valid = false;
        warp_reduce_add(E, s, e, valid);
    }
}

// contact energy at the current positions: kappa dt^2 b(x) over active pairs
__global__ void k_ee_energy(int ne, GridView GV, Geo G, const float4* __restrict__ qlo, const float4* __restrict__ qhi,
                            const int* __restrict__ qscene, int f32, int self_contact, double dhat, int barrier,
                            double sc, const int* done, double* E) {
    for (long base = (long)blockIdx.x * blockDim.x; base < ne; base += (long)gridDim.x * blockDim.x) {
        long i = base + threadIdx.x;
        bool valid = i < ne;
        int s = valid ? qscene[i] : 0;
        double e = 0;
        if (valid && !done[s]) {
            int ii = (int)i;
            double xh = dhat * dhat;
            grid_visit(GV, qlo[i], qhi[i], s, [&](int j) {
                if (j <= ii) return;
                int2 ea = G.edges[ii], eb = G.edges[j];
                if (ea.x == eb.x || ea.x == eb.y || ea.y == eb.x || ea.y == eb.y) return;
                if (!self_contact && G.vbody[ea.x] == G.vbody[eb.x]) return;
                int4 stv; int type; double xb;
                if (!classify(G, ABD_CONTACT_EE, ii, j, f32, dhat, stv, type, xb)) return;
                double b0, b1, b2; barrier3(barrier, xb, xh, b0, b1, b2);
                e += b0 * sc;
            });
        } else valid = false;
        warp_reduce_add(E, s, e, valid);
    }
}
__global__ void k_pt_energy(int nv, GridView GV, Geo G, const float4* __restrict__ qlo, const float4* __restrict__ qhi,
                            const int* __restrict__ qscene, int self_contact, double dhat, int barrier, double sc,
                            const int* done, double* E) {
    for (long base = (long)blockIdx.x * blockDim.x; base < nv; base += (long)gridDim.x * blockDim.x) {
        long p = base + threadIdx.x;
        bool valid = p < nv;
        int s = valid ? qscene[p] : 0;
        double e = 0;
        if (valid && !done[s]) {
            int pp = (int)p;
            double xh = dhat * dhat;
            grid_visit(GV, qlo[p], qhi[p], s, [&](int t) {
                int ta = G.tris[3*t];
                if (pp == ta || pp == G.tris[3*t+1] || pp == G.tris[3*t+2]) return;
                if (!self_contact && G.vbody[pp] == G.vbody[ta]) return;
                int4 stv; int type; double xb;
                if (!classify(G, ABD_CONTACT_PT, pp, t, 0, dhat, stv, type, xb)) return;
                double b0, b1, b2; barrier3(barrier, xb, xh, b0, b1, b2);
                e += b0 * sc;
            });
        } else valid = false;
        warp_reduce_add(E, s, e, valid);
    }
}
__global__ void k_pg_energy(int nv, Geo G, const int* __restrict__ vscene, PairTerms T, const int* done, double* E) {
    for (long base = (long)blockIdx.x * blockDim.x; base < nv; base += (long)gridDim.x * blockDim.x) {
        long v = base + threadIdx.x;
        bool valid = v < nv;
        int s = valid ? vscene[v] : 0;
        double e = 0, en = 0;
        if (valid && !done[s]) {
            for (int pl = G.sc_plane_begin[s]; pl < G.sc_plane_begin[s+1]; pl++) plane_energy(G.x + 3*v, G.planes + 4*pl, T, e, en);
        } else valid = false;
        warp_reduce_add(E, s, e, valid);
    }
}

// energy per scene into scd[slot]; scenes flagged in sci[SI_ACC] (accepted)
// or sci[SI_DONE] are skipped via the `skip` array argument
static int energy_impl(Engine* E, int slot, const int* skip) {
    cudaStream_t s = E->stream;
    int rc;
    double* Eo = E->scd + slot * E->ns;
    CUDA_TRY(cudaMemsetAsync(Eo, 0, sizeof(double) * E->ns, s));
    if ((rc = eng_transform(E))) return rc;
    const AbdParams& P = E->P;
    if ((rc = eng_body_energy(E, Eo, skip))) return rc;
    double sc = P.kappa * P.dt * P.dt;
    Geo G = geo(E);
    if (P.contact_ee && E->ne > 1) {
        if ((rc = build_ee_grid(E, P.dhat))) return rc;
        Grid& g = E->gee;
        int ph = phase_begin(E, PH_EQUERY);
        k_ee_energy<<<grid_for(E->ne, 128), 128, 0, s>>>(E->ne, eng_view(g), G, g.lo, g.hi, g.scene, P.ee_f32, P.self_contact,
                                                          P.dhat, P.barrier, sc, skip, Eo);
        // edges, their boxes/scene, sorted values, bucket table, positions
        phase_end(E, ph, E->ne * (8.0 + 32.0 + 4.0 + 4.0) + g.H * 8.0 + E->nv * (P.ee_f32 ? 16.0 : 24.0));
        E->launches++;
    }
    if (P.contact_pt && E->nt > 0) {
        if ((rc = build_pt_grid(E, P.dhat))) return rc;
        Grid& g = E->gpt;
        int ph = phase_begin(E, PH_EQUERY);
        k_pt_energy<<<grid_for(E->nv, 128), 128, 0, s>>>(E->nv, eng_view(g), G, g.qlo, g.qhi, g.qscene, P.self_contact, P.dhat,
                                                          P.barrier, sc, skip, Eo);
        // points and their boxes, triangles, their boxes/scene, sorted values, buckets, positions
        phase_end(E, ph, E->nv * (32.0 + 4.0 + 24.0) + E->nt * (12.0 + 32.0 + 4.0 + 4.0) + g.H * 8.0);
        E->launches++;
    }
    return eng_pg_energy(E, Eo, skip);
}
int eng_body_energy(Engine* E, double* Eo, const int* skip) {
    k_body_energy<<<grid_for(E->nb), 256, 0, E->stream>>>(E->nb, E->st, E->mass, E->J, E->bscene, body_terms(E->P), skip, Eo);
    E->launches++;
    return ABD_OK;
}
int eng_pg_energy(Engine* E, double* Eo, const int* skip) {
    if (E->npl > 0) {
        k_pg_energy<<<grid_for(E->nv), 256, 0, E->stream>>>(E->nv, geo(E), E->vscene, pair_terms(E->P), skip, Eo);
        E->launches++;
    }
    return ABD_OK;
}
int eng_energy(Engine* E, int slot) { return energy_impl(E, slot, E->sci + SI_DONE * E->ns); }
int eng_energy_masked(Engine* E, int slot, const int* skip) { return energy_impl(E, slot, skip); }

// ------------------------------------------------------------------ intersections
DV double orient3(d3 a, d3 b, d3 c, d3 d) { return dot(cross(b - a, c - a), d - a); }
__global__ void k_intersections(int ne, GridView GV, Geo G, const float4* __restrict__ qlo, const float4* __restrict__ qhi,
                                const int* __restrict__ qscene, int* count) {
    GS_LOOP(e, ne) {
        int2 ed = G.edges[e];
        d3 P = ld3(G.x + 3*ed.x), Q = ld3(G.x + 3*ed.y);
        int be = G.vbody[ed.x];
        int c = 0;
        grid_visit(GV, qlo[e], qhi[e], qscene[e], [&](int t) {
            int a = G.tris[3*t], b = G.tris[3*t+1], cc = G.tris[3*t+2];
            if (G.vbody[a] == be) return;
            d3 A = ld3(G.x + 3*a), B = ld3(G.x + 3*b), C = ld3(G.x + 3*cc);
            double o1 = orient3(A, B, C, P), o2 = orient3(A, B, C, Q);
            if ((o1 > 0 && o2 > 0) || (o1 < 0 && o2 < 0) || (o1 == 0 && o2 == 0)) return;
            double s1 = orient3(P, Q, A, B), s2 = orient3(P, Q, B, C), s3 = orient3(P, Q, C, A);
            if ((s1 > 0 && s2 > 0 && s3 > 0) || (s1 < 0 && s2 < 0 && s3 < 0)) c++;
        });
        if (c) atomicAdd(count, c);
    }
}
int eng_intersections(Engine* E, int* count) {
    *count = 0;
    if (E->nt == 0 || E->ne == 0) return ABD_OK;
    cudaStream_t s = E->stream;
    int rc;
    if ((rc = eng_transform(E))) return rc;
    Grid& g = E->gpt;   // triangles stored; edge boxes as queries (in the EE grid's box arrays)
    CUDA_TRY(cudaMemsetAsync(g.cell, 0, sizeof(float), s));
    CUDA_TRY(cudaMemsetAsync(&E->dcnt->nkeys, 0, sizeof(int), s));
    k_tri_boxes<<<grid_for(g.n), 256, 0, s>>>(g.n, E->tris, E->x, E->tri_scene, 0.f, g.lo, g.hi, g.scene, g.cell);
    Grid& q = E->gee;
    k_edge_boxes<<<grid_for(q.n), 256, 0, s>>>(q.n, E->edges, E->x, E->xf, E->edge_scene, 0.f, 0, q.lo, q.hi, q.scene, g.cell);
    if ((rc = eng_grid_build(E, g))) return rc;
    k_intersections<<<grid_for(E->ne, 128), 128, 0, s>>>(E->ne, eng_view(g), geo(E), q.lo, q.hi, q.scene, &E->dcnt->nkeys);
    E->launches += 3;
    CUDA_TRY(cudaMemcpyAsync(E->hcnt, E->dcnt, sizeof(Counters), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(eng_stream_sync(E));
    *count = E->hcnt->nkeys;
    return ABD_OK;
}

// exported for assemble.cu
Geo eng_geo(Engine* E) { return geo(E); }
