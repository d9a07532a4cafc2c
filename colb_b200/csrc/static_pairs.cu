// static_pairs.cu — edge-edge candidate detection that allocates nothing.
//
// Some callers cannot allocate device memory when they need the candidate
// pairs: a host application that has handed all device memory management to
// its own pool, a real-time loop that forbids allocation after start-up, or
// a plugin running inside a host that owns the CUDA context and bans
// cudaMalloc.  abd_ee_pairs_static serves them: the caller passes device
// buffers for its inputs and outputs, and every intermediate (boxes, grid
// keys, buckets, per-edge counts, radix-sort and scan scratch) lives in the
// file-scope __device__ arrays below, sized for ABD_STATIC_MAX_EDGES edges.
// Every GPU that loads the library holds these arrays until the process
// exits: boxes 4 MiB (by edge and by cell), grid keys 0.5 MiB, buckets 1 MiB,
// per-edge counts, offsets and list positions 0.75 MiB, partner lists 4 MiB,
// scan scratch 0.25 MiB, about 10.5 MiB in all.
//
// Host code must not pass the arrays' names to a kernel: in host code a
// __device__ symbol names a host-side stand-in, not device memory.  The
// first call on each device, with that device current, looks the device
// addresses up with cudaGetSymbolAddress and caches them; make that first
// call before any stream capture.  The cache is not refreshed: after a
// cudaDeviceReset of a device, this entry point must not be called on that
// device again in the same process.  Every call waits for its stream before
// it returns (it reads the pair count back).  All calls share the arrays:
// two calls whose work overlaps on the GPU (different streams, or the same
// arrays used by two threads at once) race and corrupt each other's results.
#include "engine.cuh"
#include "physics.cuh"
#include <cub/cub.cuh>
#include <mutex>

std::string& abd_global_error();   // capi.cu: the message abd_last_error(NULL) returns

#define ST_MAXE ABD_STATIC_MAX_EDGES
#define ST_H (2 * ST_MAXE)
#define ST_CUB_BYTES (256 << 10)
#define ST_POOL (1 << 20)                // partners that the lists of all edges hold
#define ST_LIST 96                       // partners of one edge that a list holds

static __device__ __align__(256) float4 g_st_box[4 * ST_MAXE];               // by edge: lo, hi; by cell: lo, hi
static __device__ __align__(256) uint32_t g_st_keys[2 * ST_MAXE];            // bucket, place in it
static __device__ __align__(256) int g_st_bucket[2 * (ST_H + 1) + 4];        // counts and flags (StaticFlags), starts
static __device__ __align__(256) int g_st_count[3 * (ST_MAXE + 1)];          // pairs, offsets, list positions
static __device__ __align__(256) int g_st_pool[ST_POOL];
static __device__ __align__(256) unsigned char g_st_cub[ST_CUB_BYTES];

struct StaticFlags { float cell; int bad; int pooled; int pad; };            // cell edge; bad edge index; pool entries taken
struct StaticScratch {
    float4* box; uint32_t* keys; int* bucket; int* count; int* pool; void* cub;
    bool ready;
};
static StaticScratch g_scratch[64];
static std::mutex g_scratch_mu;

static int scratch_for_device(int dev, StaticScratch** out, std::string& err) {
    if (dev < 0 || dev >= 64) { err = "abd_ee_pairs_static: device index out of range"; return ABD_ERR_INVALID_ARG; }
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    StaticScratch& S = g_scratch[dev];
    if (!S.ready) {
        struct { void** p; const void* sym; } t[] = {
            {(void**)&S.box, (const void*)&g_st_box}, {(void**)&S.keys, (const void*)&g_st_keys},
            {(void**)&S.bucket, (const void*)&g_st_bucket}, {(void**)&S.count, (const void*)&g_st_count},
            {(void**)&S.pool, (const void*)&g_st_pool}, {(void**)&S.cub, (const void*)&g_st_cub}};
        for (auto& e : t) {
            cudaError_t rc = cudaGetSymbolAddress(e.p, e.sym);
            if (rc != cudaSuccess) {
                err = std::string("abd_ee_pairs_static: cudaGetSymbolAddress: ") + cudaGetErrorString(rc);
                return ABD_ERR_CUDA;
            }
        }
        S.ready = true;
    }
    *out = &S;
    return ABD_OK;
}

// boxes of the float32 copies of the endpoints (contact.py:150-154), padded.
// Every edge index must name a vertex of x: one that does not sets F->bad, and
// the kernels after this one do nothing.
__global__ void k_st_boxes(int ne, int nv, const double* __restrict__ x, const int* __restrict__ edges, float pad,
                           float4* lo, float4* hi, StaticFlags* F) {
    float ext = 0.f;
    GS_LOOP(e, ne) {
        int a = edges[2*e], b = edges[2*e+1];
        if ((unsigned)a >= (unsigned)nv || (unsigned)b >= (unsigned)nv) { F->bad = 1; continue; }
        float l[3], h[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float fa = __double2float_rn(x[3*a+k]), fb = __double2float_rn(x[3*b+k]);
            l[k] = __fsub_rd(fminf(fa, fb), pad); h[k] = __fadd_ru(fmaxf(fa, fb), pad);
        }
        lo[e] = make_float4(l[0], l[1], l[2], 0.f); hi[e] = make_float4(h[0], h[1], h[2], 0.f);
        ext = fmaxf(ext, fmaxf(h[0] - l[0], fmaxf(h[1] - l[1], h[2] - l[2])));
    }
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if ((threadIdx.x & 31) == 0 && ext > 0.f) atomic_max_pos(&F->cell, ext);
}
// The edges are put in order of their buckets by counting: an edge's place in
// its bucket is the count it found there (k_st_keys), a bucket's start the sum
// of the counts below it, and k_st_fill copies the boxes to their places, so a
// query reads a bucket's boxes from consecutive addresses.  The order within a
// bucket is not fixed; the order of the results does not depend on it.  (A
// radix sort of the keys took 45 us for 55,296 edges.)
__global__ void k_st_keys(int n, const float4* __restrict__ lo, const StaticFlags* F, uint32_t mask, uint32_t* key,
                          uint32_t* place, int* bucket) {
    if (F->bad) return;
    float h = fmaxf(F->cell, 1e-6f);
    GS_LOOP(i, n) {
        float4 l = lo[i];
        uint32_t k = cell_hash(0, (int)floorf(l.x / h), (int)floorf(l.y / h), (int)floorf(l.z / h)) & mask;
        key[i] = k;
        place[i] = atomicAdd(bucket + k, 1);
    }
}
// boxes in bucket order, the edge in lo's fourth word
__global__ void k_st_fill(int n, const float4* __restrict__ lo, const float4* __restrict__ hi, const StaticFlags* F,
                          const uint32_t* __restrict__ key, const uint32_t* __restrict__ place,
                          const int* __restrict__ start, float4* lo_s, float4* hi_s) {
    if (F->bad) return;
    GS_LOOP(i, n) {
        int at = start[key[i]] + (int)place[i];
        float4 l = lo[i];
        l.w = __int_as_float((int)i);
        lo_s[at] = l; hi_s[at] = hi[i];
    }
}

struct StaticGrid {
    const float4 *lo, *hi;               // by edge
    const float4 *lo_s, *hi_s;           // by bucket
    const int* start;                    // bucket k: [start[k], start[k + 1])
    uint32_t mask;
    const double* x; const int* edges;
    float cand;
};
// One warp visits the partners j > i of edge i closer than cand: emit(found, j)
// is called by all lanes together, with the lane's j where found.  The lanes
// look up 32 cells at once and then take the items of all of them side by side
// (a lane finds the cell of its item by bisecting the running sums), and the
// boxes that overlap wait in `queue` (64 ints of the warp's shared memory)
// until 32 segment distances can be computed at once.
template <class F>
DV void st_visit(const StaticGrid& G, float h, int i, int* queue, F&& emit) {
    const int lane = threadIdx.x & 31;
    const float4 qlo = G.lo[i], qhi = G.hi[i];
    const int a0 = G.edges[2*i], a1 = G.edges[2*i+1];
    int c0[3], c1[3];
    if (!grid_range(h, qlo, qhi, c0, c1)) return;
    const int nx = c1[0] - c0[0] + 1, ny = c1[1] - c0[1] + 1, ncell = nx * ny * (c1[2] - c0[2] + 1);
    float p1[3], q1[3];
    for (int k = 0; k < 3; k++) { p1[k] = __double2float_rn(G.x[3*a0+k]); q1[k] = __double2float_rn(G.x[3*a1+k]); }
    int queued = 0;
    auto flush = [&](int n) {            // the first n <= 32 of the queue
        bool found = lane < n;
        int j = found ? queue[lane] : 0;
        if (found) {
            int b0 = G.edges[2*j], b1 = G.edges[2*j+1];
            found = !(a0 == b0 || a0 == b1 || a1 == b0 || a1 == b1);
            if (found) {
                float p2[3], q2[3];
                for (int k = 0; k < 3; k++) { p2[k] = __double2float_rn(G.x[3*b0+k]); q2[k] = __double2float_rn(G.x[3*b1+k]); }
                float s, t, d;
                seg_seg_f32(p1, q1, p2, q2, 1e-6f, s, t, d);
                found = d < G.cand;
            }
        }
        emit(found, j);
        __syncwarp();
    };
    for (int cb = 0; cb < ncell; cb += 32) {
        int cell = cb + lane, b = 0, n = 0;
        const int cx = c0[0] + cell % nx, cy = c0[1] + cell / nx % ny, cz = c0[2] + cell / (nx * ny);
        if (cell < ncell) {
            const uint32_t key = cell_hash(0, cx, cy, cz) & G.mask;
            b = G.start[key]; n = G.start[key + 1] - b;
        }
        int sum = n;                     // items of this lane's cell and the ones before it
        for (int o = 1; o < 32; o <<= 1) { int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
        const int total = __shfl_sync(0xffffffffu, sum, 31);
        for (int f0 = 0; f0 < total; f0 += 32) {
            const int f = f0 + lane;
            int c = 0;                   // the first lane whose sum exceeds f
            for (int o = 16; o > 0; o >>= 1) c += __shfl_sync(0xffffffffu, sum, c + o - 1) <= f ? o : 0;
            const int at = __shfl_sync(0xffffffffu, b + n - sum, c) + f;
            const int kx = __shfl_sync(0xffffffffu, cx, c), ky = __shfl_sync(0xffffffffu, cy, c), kz = __shfl_sync(0xffffffffu, cz, c);
            bool in = f < total;
            int j = 0;
            if (in) {
                const float4 lo = G.lo_s[at];
                j = __float_as_int(lo.w);
                // a bucket can hold other cells' items; they are visited from their own cell
                in = j > i && boxes_overlap(lo, G.hi_s[at], qlo, qhi) && (int)floorf(lo.x / h) == kx &&
                     (int)floorf(lo.y / h) == ky && (int)floorf(lo.z / h) == kz;
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) queue[queued + __popc(m & ((1u << lane) - 1))] = j;
            __syncwarp();
            queued += __popc(m);
            if (queued >= 32) {
                flush(32);
                queued -= 32;
                const int v = lane < queued ? queue[32 + lane] : 0;
                __syncwarp();
                if (lane < queued) queue[lane] = v;
                __syncwarp();
            }
        }
    }
    if (queued > 0) flush(queued);
}
// Counts each edge's pairs and keeps its partners, in order, at pool[at[i]].  at[i] = -1:
// more partners than ST_LIST or than the pool has room for (k_st_write visits again).  One warp
// per edge: with one thread per edge, a count pass and a write pass of the
// same walk took 609 us each for 55,296 edges (245 boxes and 13 distances per
// edge); this pass takes 117 us, the write 17.
__global__ void __launch_bounds__(256) k_st_find(int ne, StaticGrid G, StaticFlags* F, int* count, int* at, int* pool) {
    __shared__ int s_queue[8][64], s_list[8][ST_LIST];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* list = s_list[w];
    if (F->bad) { if (threadIdx.x == 0 && blockIdx.x == 0) count[ne] = 0; return; }
    const float h = F->cell;
    for (int i = blockIdx.x * 8 + w; i <= ne; i += gridDim.x * 8) {
        if (i == ne) { if (lane == 0) count[ne] = 0; break; }
        int c = 0;
        st_visit(G, h, i, s_queue[w], [&](bool found, int j) {
            const unsigned m = __ballot_sync(0xffffffffu, found);
            const int k = c + __popc(m & ((1u << lane) - 1));
            if (found && k < ST_LIST) list[k] = j;
            c += __popc(m);
        });
        __syncwarp();
        int base = -1;
        if (lane == 0) {
            count[i] = c;
            if (c > 0 && c <= ST_LIST) {
                base = atomicAdd(&F->pooled, c);
                if (base + c > ST_POOL) base = -1;
            }
            at[i] = base;
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= 0)
            for (int k = lane; k < c; k += 32) {
                const int j = list[k];
                int rank = 0;
                for (int l = 0; l < c; l++) rank += list[l] < j;
                pool[base + rank] = j;
            }
        __syncwarp();
    }
}
// Writes vertex quadruples, by edge and partner, the rows that fit below cap.
// An edge without a list (see k_st_find) visits its partners again and orders
// them where they are written.  The order of a visit is not fixed (k_st_keys),
// so the one edge whose rows may cross cap keeps its smallest partners, each
// put in its place as it is found: the rows are the first ones of the complete list.
__global__ void __launch_bounds__(256) k_st_write(int ne, StaticGrid G, const StaticFlags* F, const int* __restrict__ count,
                                                  const int* __restrict__ off, const int* __restrict__ at,
                                                  const int* __restrict__ pool, int* out4, int cap, int* n_out) {
    __shared__ int s_queue[8][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (F->bad) return;
    const float h = F->cell;
    if (threadIdx.x == 0 && blockIdx.x == 0) *n_out = off[ne];
    for (int i = blockIdx.x * 8 + w; i < ne; i += gridDim.x * 8) {
        const int c = count[i], base = off[i], from = at[i];
        if (c == 0 || base >= cap) continue;
        const int rows = min(c, cap - base);
        if (from < 0 && rows < c) {
            int have = 0;                                    // lane 0's: rows so far, in order
            st_visit(G, h, i, s_queue[w], [&](bool found, int j) {
                for (unsigned m = __ballot_sync(0xffffffffu, found); m; m &= m - 1) {
                    const int v = __shfl_sync(0xffffffffu, j, __ffs(m) - 1);
                    if (lane > 0 || (have == rows && out4[4L*(base+rows-1)+2] < v)) continue;
                    int k = base + (have < rows ? have++ : rows - 1);
                    for (; k > base && out4[4L*(k-1)+2] > v; k--) out4[4L*k+2] = out4[4L*(k-1)+2];
                    out4[4L*k+2] = v;
                }
            });
            __syncwarp();
        } else if (from < 0) {
            int k0 = base;
            st_visit(G, h, i, s_queue[w], [&](bool found, int j) {
                const unsigned m = __ballot_sync(0xffffffffu, found);
                const int k = k0 + __popc(m & ((1u << lane) - 1));
                if (found && k < cap) out4[4L*k+2] = j;
                k0 += __popc(m);
            });
            __syncwarp();
            if (lane == 0)
                for (int k = base + 1; k < base + rows; k++) {
                    int j = out4[4L*k+2], m = k - 1;
                    while (m >= base && out4[4L*m+2] > j) { out4[4L*(m+1)+2] = out4[4L*m+2]; m--; }
                    out4[4L*(m+1)+2] = j;
                }
            __syncwarp();
        }
        for (int k = lane; k < rows; k += 32) {
            int* o = out4 + 4L * (base + k);
            const int j = from < 0 ? o[2] : pool[from + k];
            o[0] = G.edges[2*i]; o[1] = G.edges[2*i+1]; o[2] = G.edges[2*j]; o[3] = G.edges[2*j+1];
        }
    }
}

extern "C" int abd_ee_pairs_static(const double* x_dev, const int32_t* edges_dev, int32_t n_verts, int32_t n_edges,
                                   double cand_dist, int32_t* pairs_dev, int32_t cap, int32_t* n_pairs_dev,
                                   void* stream_ptr) {
    std::string& err = abd_global_error();
    if (n_edges < 0 || n_verts < 0 || n_edges > ST_MAXE || cap < 0 || !(cand_dist > 0) ||
        (n_edges > 0 && (!x_dev || !edges_dev)) || !n_pairs_dev || (cap > 0 && !pairs_dev)) {
        err = "abd_ee_pairs_static: invalid arguments (n_edges must be in [0, " + std::to_string(ST_MAXE) +
              "], cand_dist > 0, device buffers non-null)";
        return ABD_ERR_INVALID_ARG;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { err = "abd_ee_pairs_static: no current device"; return ABD_ERR_NO_DEVICE; }
    StaticScratch* S = nullptr;
    int rc = scratch_for_device(dev, &S, err);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream_ptr;
    if (n_edges < 2) {
        if (cudaMemsetAsync(n_pairs_dev, 0, sizeof(int32_t), s) != cudaSuccess) { err = "abd_ee_pairs_static: cudaMemsetAsync failed"; return ABD_ERR_CUDA; }
        return cudaStreamSynchronize(s) == cudaSuccess ? ABD_OK : ABD_ERR_CUDA;
    }
    int H = 64; while (H < 2 * n_edges) H <<= 1;
    float pad = (float)(0.5 * cand_dist * (1.0 + 1e-6) + 1e-7);
    float4 *lo = S->box, *hi = lo + ST_MAXE, *lo_s = hi + ST_MAXE, *hi_s = lo_s + ST_MAXE;
    uint32_t *key = S->keys, *place = key + ST_MAXE;
    StaticFlags* F = (StaticFlags*)S->bucket;
    int *bcount = S->bucket + 4, *bstart = bcount + ST_H + 1;
    int *count = S->count, *off = count + ST_MAXE + 1, *at = off + ST_MAXE + 1;
    size_t need = 0, need2 = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, need, bcount, bstart, H + 1, s);
    cub::DeviceScan::ExclusiveSum(nullptr, need2, count, off, n_edges + 1, s);
    if (need > ST_CUB_BYTES || need2 > ST_CUB_BYTES) { err = "abd_ee_pairs_static: scan scratch exceeds the static size"; return ABD_ERR_INVALID_ARG; }
    // clear what the previous call left behind: the flags and the bucket counts, one range
    if (cudaMemsetAsync(F, 0, sizeof(StaticFlags) + sizeof(int) * (H + 1), s) != cudaSuccess ||
        cudaMemsetAsync(n_pairs_dev, 0, sizeof(int32_t), s) != cudaSuccess) {
        err = "abd_ee_pairs_static: cudaMemsetAsync failed"; return ABD_ERR_CUDA;
    }
    k_st_boxes<<<grid_for(n_edges), 256, 0, s>>>(n_edges, n_verts, x_dev, edges_dev, pad, lo, hi, F);
    k_st_keys<<<grid_for(n_edges), 256, 0, s>>>(n_edges, lo, F, (uint32_t)(H - 1), key, place, bcount);
    if (cub::DeviceScan::ExclusiveSum(S->cub, need, bcount, bstart, H + 1, s) != cudaSuccess) {
        err = "abd_ee_pairs_static: scan failed"; return ABD_ERR_CUDA;
    }
    k_st_fill<<<grid_for(n_edges), 256, 0, s>>>(n_edges, lo, hi, F, key, place, bstart, lo_s, hi_s);
    StaticGrid G{lo, hi, lo_s, hi_s, bstart, (uint32_t)(H - 1), x_dev, edges_dev, (float)cand_dist};
    k_st_find<<<grid_for(32L * n_edges), 256, 0, s>>>(n_edges, G, F, count, at, S->pool);
    if (cub::DeviceScan::ExclusiveSum(S->cub, need2, count, off, n_edges + 1, s) != cudaSuccess) {
        err = "abd_ee_pairs_static: scan failed"; return ABD_ERR_CUDA;
    }
    k_st_write<<<grid_for(32L * n_edges), 256, 0, s>>>(n_edges, G, F, count, off, at, S->pool, pairs_dev, cap, n_pairs_dev);
    int bad = 0;
    if (cudaMemcpyAsync(&bad, &F->bad, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) { err = "abd_ee_pairs_static: CUDA error"; return ABD_ERR_CUDA; }
    int n = 0;
    if (cudaMemcpyAsync(&n, n_pairs_dev, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        err = std::string("abd_ee_pairs_static: ") + cudaGetErrorString(cudaGetLastError());
        return ABD_ERR_CUDA;
    }
    if (bad) { err = "abd_ee_pairs_static: an edge index is outside [0, n_verts)"; return ABD_ERR_INVALID_ARG; }
    if (n > cap) { err = "abd_ee_pairs_static: more pairs than cap (the count is in *n_pairs_dev)"; return ABD_ERR_CONTACT_OVERFLOW; }
    return ABD_OK;
}
