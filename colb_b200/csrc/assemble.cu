// assemble.cu — gradient and block Hessian of the incremental potential.
//
//  inertia + orthogonality  abd.py:108-166, ortho.py:9-41 (one warp per body, one thread its SVD)
//  barrier contacts ....... abd.py:198-571: classify each candidate into a
//                           PP / PE / EE (or PT / PG) stencil, differentiate its
//                           squared distance, chain through the barrier and map
//                           vertex derivatives to body DoFs with
//                           J = [1, xbar^T] (x) I3.
//
// The reference writes 64 triplets per contact into a COO array (with the
// contact/inertia slot overlap at abd.py:111 vs :311) and converts the whole
// array to BSR every iteration (abd.py:634).  Here the body-pair pattern is
// built once per Newton iteration from bits that the contacts set (k_bit_rows:
// CSR of 12x12 blocks; a radix sort of 64-bit body-pair keys where the bits
// would take too many words), and each active
// contact adds its four body blocks into that structure with FP64/FP32
// atomics.
#include "contact.cuh"
#include "contact_hess.cuh"
#include "block_inverse.cuh"
#include <cub/cub.cuh>

Geo eng_geo(Engine* E);

DV int stencil_np(int type) { return type == T_PP ? 2 : (type == T_PE ? 3 : (type == T_PG ? 1 : 4)); }
DV int other_vertex(int type, int4 s) { return type == T_EE ? s.z : (type == T_PG ? s.x : s.y); }

// ---------------------------------------------------------- prepare + keys
// Pattern of the block rows as bits: row b has `words` words, bit c for
// body c of its scene (null: the keys below instead).  k_bit_rows clears what it reads.
struct BitRows { uint32_t* bits; int words; const int* bscene; const int* sc_body_begin; };
DV void set_bit(const BitRows& B, int r, int c) {
    uint32_t* w = B.bits + (long)r * B.words + (c >> 5);
    const uint32_t m = 1u << (c & 31);
    if (!(*(volatile uint32_t*)w & m)) atomicOr(w, m);
}
// Contacts [0, n_total) (the device count, at most cap); with nkey_pairs > n_total the key
// pairs of the slots up to nkey_pairs are sentinels (~0), so a sort sized
// before the count is known sees only real keys and sentinels.
__global__ void k_contact_prepare(const Counters* cnt, const int4* __restrict__ contacts, Geo G, int f32, double dhat,
                                  int nb, int cap, int4* cst, int* ctype, double* cxb, int2* cbody,
                                  unsigned long long* keys, BitRows B, int* n_active, int nkey_pairs) {
    int n = min(cnt->n_total, cap);
    if (!B.bits) GS_LOOP(c, nkey_pairs) {
        if (c >= n) { keys[nb + 2*c] = ~0ull; keys[nb + 2*c + 1] = ~0ull; }
    }
    GS_LOOP(c, n) {
        int4 C = contacts[c];
        int4 stv; int type = -1; double xb = 0;
        bool act = classify(G, C.x, C.y, C.z, f32, dhat, stv, type, xb);
        unsigned long long k0 = ~0ull, k1 = ~0ull;
        if (act) {
            int b0 = G.vbody[stv.x];
            int b1 = G.vbody[other_vertex(type, stv)];
            cbody[c] = make_int2(b0, b1);
            if (b0 != b1 && G.mass[b0] > 0.0 && G.mass[b1] > 0.0) {
                if (B.bits) {
                    const int f = B.sc_body_begin[B.bscene[b0]];
                    set_bit(B, b0, b1 - f); set_bit(B, b1, b0 - f);
                }
                k0 = (unsigned long long)b0 * nb + b1;
                k1 = (unsigned long long)b1 * nb + b0;
            }
            atomicAdd(n_active, 1);
        }
        cst[c] = stv; ctype[c] = act ? type : -1; cxb[c] = xb;
        if (!B.bits) { keys[nb + 2*c] = k0; keys[nb + 2*c + 1] = k1; }
    }
}
// Block rows from the bits, by one block or, from BR_SPLIT words on, a cluster of eight, each
// with a run of rows: each row's count, their running
// sums, then the columns (ascending, so this is the order a sort of the keys
// gives).  A row is read by `lanes` threads, a power of two up to a warp, one
// word each.  The bits and the contact count are cleared for the next
// assembly, and what the host's component analysis reads is written to its pinned
// memory from here.  Replaces clearing, diagonal keys, a radix sort, the
// removal of doubles, the rows and three copies, 38 us of an iteration of eight
// cubes: 7 us now; 10 for the 256 bodies of a net, 18 for 512 scenes of 10,801
// bodies (one block for those: 69).
constexpr int BR_CL = 8, BR_SPLIT = 4096;
DV uint32_t br_cluster_blocks() { uint32_t n; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n)); return n; }
DV uint32_t br_cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
DV void br_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
DV void br_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// v to `p` of this block's shared memory in block `rank` of the cluster
DV void br_store(int* p, int rank, int v) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}
struct BitHost { int* row; int* col; int* done; Counters* cnt; };      // null: not wanted
__global__ void __launch_bounds__(1024) k_bit_rows(int nb, int bound, BitRows B, int lanes, int* row_ptr, int* bcol,
                                                   Counters* cnt, int ns, const int* done, BitHost H) {
    __shared__ int s_sum[32], s_of[BR_CL];
    __shared__ int s_total;
    const uint32_t C = br_cluster_blocks(), c = br_cluster_rank();
    // the other blocks' shared memory may be written once they all run: they
    // meet here, and the wait comes after the rows are counted
    if (C > 1) br_cluster_arrive();
    const int share = (nb + (int)C - 1) / (int)C, b0 = min((int)c * share, nb), b1 = min(b0 + share, nb);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = tid & (lanes - 1);
    const unsigned group = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1) << (lane & ~(lanes - 1));
#pragma unroll 4
    for (int r = b0 + tid / lanes; r < b1; r += 1024 / lanes) {
        const int self = r - B.sc_body_begin[B.bscene[r]];
        int n = 0;
        for (int w = sub; w < B.words; w += lanes) {
            uint32_t v = B.bits[(long)r * B.words + w];
            if (w == self >> 5) v |= 1u << (self & 31);
            n += __popc(v);
        }
        for (int o = lanes / 2; o > 0; o >>= 1) n += __shfl_xor_sync(group, n, o);
        if (sub == 0) row_ptr[r] = n;
    }
    __syncthreads();
    // exclusive sums, each thread over a run of rows
    const int per = (b1 - b0 + 1023) / 1024, r0 = min(b0 + tid * per, b1), r1 = min(r0 + per, b1);
    int mine = 0;
    for (int r = r0; r < r1; r++) mine += row_ptr[r];
    int incl = mine;
    for (int o = 1; o < 32; o <<= 1) { int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int v = s_sum[lane];
        for (int o = 1; o < 32; o <<= 1) { int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        if (lane == 31) s_total = v;
        s_sum[lane] = v - s_sum[lane];
    }
    __syncthreads();
    int before = 0, all = s_total;           // blocks of the rows of the cluster's earlier blocks, of all rows
    if (C > 1) {
        br_cluster_wait();
        if (tid < (int)C) br_store(&s_of[c], tid, s_total);
        br_cluster_arrive();
        br_cluster_wait();
        all = 0;
        for (int k = 0; k < (int)C; k++) { if (k < (int)c) before += s_of[k]; all += s_of[k]; }
    }
    for (int r = r0, at = before + s_sum[warp] + incl - mine; r < r1; r++) { const int n = row_ptr[r]; row_ptr[r] = at; at += n; }
    if (tid == 0 && c == 0) {
        row_ptr[nb] = all;
        if (H.row) H.row[nb] = all;
        cnt->nnzb = cnt->nkeys = all;
        cnt->n_active = cnt->act; cnt->act = 0;
    }
    __syncthreads();
#pragma unroll 2
    for (int r = b0 + tid / lanes; r < b1; r += 1024 / lanes) {
        const int first = B.sc_body_begin[B.bscene[r]], self = r - first;
        int base = row_ptr[r];
        for (int w0 = 0; w0 < B.words; w0 += lanes) {
            const int w = w0 + sub;
            uint32_t v = 0;
            if (w < B.words) {
                uint32_t* p = B.bits + (long)r * B.words + w;
                v = *p;
                if (v) *p = 0;
                if (w == self >> 5) v |= 1u << (self & 31);
            }
            int n = __popc(v), sum = n;
            for (int o = 1; o < lanes; o <<= 1) { int u = __shfl_up_sync(group, sum, o, lanes); if (sub >= o) sum += u; }
            for (int at = base + sum - n; v; v &= v - 1, at++) {
                if (at >= bound) break;              // a count beyond the host's guess: it will assemble again
                bcol[at] = first + 32 * w + __ffs(v) - 1;
            }
            base += __shfl_sync(group, sum, lanes - 1, lanes);
        }
    }
    __syncthreads();
    // whole lines at a time: single words took 60 us for 4,096 rows
    if (H.row) {
        const int m = min(before + s_total, bound);
        for (int i = b0 + tid; i < b1; i += 1024) H.row[i] = row_ptr[i];
        for (int i = before + tid; i < m; i += 1024) H.col[i] = bcol[i];
    }
    if (c > 0) return;
    if (H.done) for (int s = tid; s < ns; s += 1024) H.done[s] = done[s];
    if (H.cnt) for (int i = tid; i < (int)(sizeof(Counters) / sizeof(int)); i += 1024) ((int*)H.cnt)[i] = ((const int*)cnt)[i];
}
__global__ void k_diag_keys(int nb, unsigned long long* keys) {
    GS_LOOP(b, nb) keys[b] = (unsigned long long)b * nb + b;
}
__global__ void k_block_rows(int nb, const unsigned long long* __restrict__ ukeys, const int* n_unique,
                             int* row_ptr, int* bcol, Counters* cnt) {
    int m = *n_unique;
    if (m > 0 && ukeys[m-1] == ~0ull) m--;            // drop the sentinel
    GS_LOOP(i, m) {
        unsigned long long k = ukeys[i];
        int r = (int)(k / nb);
        bcol[i] = (int)(k % nb);
        if (i == 0 || (int)(ukeys[i-1] / nb) != r) row_ptr[r] = (int)i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { row_ptr[nb] = m; cnt->nnzb = m; }
}


// ---------------------------------------------------- inertia + ortho (abd.py:108-149)
// A block takes `per` bodies.  When the Hessian is projected to PSD, one
// thread per body first computes the SVD of its affine matrix (thousands of
// dependent operations, the same for every lane if a warp did it).  Then one
// warp per body: gradient by lanes 0..11, the 9x9 orthogonality Hessian
// (scaled by dt^2) built lane-parallel in shared memory and written with the
// mass terms into the diagonal block; the warp also clears the row's other
// blocks for the contacts.  `per` is a warp's body each while there are
// multiprocessors for all blocks (the latency of one SVD bounds it then), and
// 32 in large batches: 10,801 bodies 23 us (one SVD per lane 55), 256
// bodies 9.9 (9.4).
#define BA_WARPS 8
#define BA_PER 32
inline int ba_per(int nb) { return nb <= 2 * NUM_SMS * BA_WARPS ? BA_WARPS : BA_PER; }
template <class T>
__global__ void __launch_bounds__(32 * BA_WARPS) k_body_assemble(int nb, int per, const double* __restrict__ st,
                                const double* __restrict__ mass, const double* __restrict__ J, double dt, double g0,
                                double g1, double g2, double k_ortho, int project, double pinned_diag,
                                const int* __restrict__ row_ptr, const int* __restrict__ bcol, T* vals, double* grad) {
    __shared__ double sA[BA_WARPS][108];       // 9 x 9, leading dimension 12
    __shared__ double sv[BA_WARPS][81];
    __shared__ double sq[BA_WARPS][9];
    __shared__ OrthoSvd usv[BA_PER];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* A = sA[w];
    const int first = blockIdx.x * per, last = min(first + per, nb);
    if (project) {
        const int b = first + (int)threadIdx.x;
        if ((int)threadIdx.x < per && b < last && mass[b] > 0.0) {
            double q[9], U[9], s[3], V[9];
#pragma unroll
            for (int k = 0; k < 9; k++) q[k] = st[ST_STRIDE * (long)b + ST_NXT + ST_Q + k];
            svd3(q, U, s, V);
            OrthoSvd& o = usv[threadIdx.x];
#pragma unroll
            for (int k = 0; k < 9; k++) { o.U[k] = U[k]; o.V[k] = V[k]; }
#pragma unroll
            for (int k = 0; k < 3; k++) o.s[k] = s[k];
        }
        __syncthreads();
    }
    for (int b = first + w; b < last; b += BA_WARPS) {
        int bi = find_block(row_ptr, bcol, b, b);
        if (bi < 0) continue;                              // every row holds its diagonal key
        T* V = vals + (long)bi * 144;
        for (int k = row_ptr[b]; k < row_ptr[b + 1]; k++)
            if (k != bi) for (int e = lane; e < 144; e += 32) vals[(long)k * 144 + e] = (T)0;
        double* g = grad + 12L * b;
        double m = mass[b];
        if (!(m > 0.0)) {
            if (lane < 12) g[lane] = 0.0;
            for (int e = lane; e < 144; e += 32) V[e] = (T)((e % 12 == e / 12) ? pinned_diag : 0.0);
            continue;
        }
        const double* now = st + ST_STRIDE * (long)b + ST_NOW; const double* nx = st + ST_STRIDE * (long)b + ST_NXT;
        if (lane < 9) sq[w][lane] = nx[ST_Q + lane];
        __syncwarp();
        const double* q = sq[w];
        double Jb = J[b];
        if (lane < 3) {
            double gv = lane == 0 ? g0 : (lane == 1 ? g1 : g2);
            double ct = now[ST_C + lane] + dt * now[ST_V + lane] + dt * dt * gv;
            g[lane] = (nx[ST_C + lane] - ct) * m;
        } else if (lane < 12) {
            int r = lane - 3, i = r / 3, c = r % 3;
            double gi = -q[3*i+c];
            for (int j = 0; j < 3; j++) gi += (q[3*i]*q[3*j] + q[3*i+1]*q[3*j+1] + q[3*i+2]*q[3*j+2]) * q[3*j+c];
            double qt = now[ST_Q + r] + dt * now[ST_QD + r];
            g[lane] = dt * dt * (gi * 4.0 * k_ortho) + (q[r] - qt) * Jb;
        }
        if (project) {
            ortho_hess_psd_warp(usv[b - first], k_ortho * dt * dt, sv[w], A, lane);    // analytic eigensystem
        } else {
            for (int e = lane; e < 81; e += 32) {
                int rr = e / 9, cc = e % 9;
                A[rr*12 + cc] = ortho_hess(q, k_ortho, rr / 3, cc / 3, rr % 3, cc % 3) * dt * dt;
            }
        }
        __syncwarp();
        for (int e = lane; e < 144; e += 32) {
            int row = e % 12, col = e / 12;
            double v;
            if (row < 3 || col < 3) v = (row == col) ? m : 0.0;
            else v = A[(row-3)*12 + (col-3)] + (row == col ? Jb : 0.0);
            V[e] = (T)v;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------- contacts (abd.py:198-571)
// A warp takes `per` contacts.  First groups of 32 / per lanes form one
// contact each: its stencil's five directions and its 5 x 5 matrix
// (contact_hess.cuh, every lane of a group the same numbers, so there is
// nothing to exchange).  Then the whole warp adds one contact after the other
// to the body blocks: the directions map to body DoFs through
// J = [1, xbar^T] (x) I3 as U_p, and block (a, b) is U_a M U_b^T.
// The time is the latency of the eigenproblem's dependent rotations, so `per`
// grows only once there are more contacts than warps that run at a time.
// 147 contacts of the resting 16 x 16 net: 87 -> 28 us per launch against one
// warp (or block) per contact with a 12 x 12 Jacobi over its lanes; 1,176
// contacts of eight nets 114 -> 40 us.
constexpr int CA_PER = 8;
struct ContactSmem {
    double m[CA_PER][15], frame[CA_PER][9], w[CA_PER][12], gd[CA_PER], J[4][4];
    int v[CA_PER][4], type[CA_PER];
    double U[2][5][12], Z[2][5][12];
};

template <class T, int CAW>
__global__ void __launch_bounds__(32 * CAW) k_contact_assemble(const Counters* cnt, const int4* __restrict__ cst,
                                   const int* __restrict__ ctype, const double* __restrict__ cxb, Geo G, int barrier,
                                   double dhat, double sc, int hess_mode, int per, const int* __restrict__ row_ptr,
                                   const int* __restrict__ bcol, T* vals, double* grad) {
    __shared__ ContactSmem sm[CAW];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ContactSmem& C = sm[w];
    const int n = cnt->n_total;
    for (int base = (blockIdx.x * CAW + w) * per; base < n; base += gridDim.x * CAW * per) {
        const int span = 32 / per, mine = lane / span, c = base + mine;
        int type = -1;
        if (mine < per && c < n) type = ctype[c];
        if (type >= 0) {
            const int4 s4 = cst[c];
            const int sv[4] = {s4.x, s4.y, s4.z, s4.w};
            const int np = stencil_np(type);
            d3 x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = i < np ? ld3(G.x + 3L * sv[i]) : mk3(0, 0, 0);
            Stencil5 S;
            stencil_hessian(type, x, type == T_PG ? G.planes + 4L * sv[1] : nullptr, S);
            double B0, B1, B2;
            barrier3(barrier, cxb[c], dhat * dhat, B0, B1, B2);
            contact_matrix5(type, hess_mode == ABD_HESS_PROJECTED, B1, B2, S);
            if (lane % span == 0) {
#pragma unroll
                for (int i = 0; i < 15; i++) C.m[mine][i] = S.a[i] * sc;
#pragma unroll
                for (int i = 0; i < 3; i++) { C.frame[mine][i] = S.n[i]; C.frame[mine][3 + i] = S.e1[i]; C.frame[mine][6 + i] = S.e2[i]; }
#pragma unroll
                for (int i = 0; i < 4; i++) { C.w[mine][i] = S.c[i]; C.w[mine][4 + i] = S.b2[i]; C.w[mine][8 + i] = S.b3[i]; C.v[mine][i] = sv[i]; }
                C.gd[mine] = 2.0 * S.d * S.cn * B1 * sc;
            }
        }
        if (mine < per && lane % span == 0) C.type[mine] = type;
        __syncwarp();
        for (int q = 0; q < per; q++) {
            const int tq = C.type[q];
            if (tq < 0) continue;                         // warp-uniform
            const int np = stencil_np(tq);
            // bodies of the (at most two) sides
            int vb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) vb[i] = i < np ? G.vbody[C.v[q][i]] : -1;
            int ba = vb[0], bb = -1;
#pragma unroll
            for (int i = 3; i > 0; i--) if (i < np && vb[i] != ba) bb = vb[i];
            const bool da = G.mass[ba] > 0.0, db = bb >= 0 && G.mass[bb] > 0.0;
            if (lane < 16) {
                const int i = lane >> 2, k = lane & 3;
                C.J[i][k] = i < np ? (k == 0 ? 1.0 : G.xbar[3L * C.v[q][i] + k - 1]) : 0.0;
            }
            __syncwarp();
            // U_p of both bodies, and Z = M U
            if (lane < 24) {
                const int side = lane / 12, row = lane % 12, al = row / 3, r = row % 3, body = side ? bb : ba;
                double sc_ = 0, s2 = 0, s3 = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) if (i < np && vb[i] == body) {
                    sc_ += C.J[i][al] * C.w[q][i]; s2 += C.J[i][al] * C.w[q][4 + i]; s3 += C.J[i][al] * C.w[q][8 + i];
                }
                const double u[5] = {sc_ * C.frame[q][r], s2 * C.frame[q][r], s3 * C.frame[q][r], sc_ * C.frame[q][3 + r], sc_ * C.frame[q][6 + r]};
#pragma unroll
                for (int p = 0; p < 5; p++) {
                    double z = 0;
#pragma unroll
                    for (int k = 0; k < 5; k++) z += C.m[q][s5(p, k)] * u[k];
                    C.U[side][p][row] = u[p]; C.Z[side][p][row] = z;
                }
                // gradient: 2 d |c| B1 along the first direction
                if (side ? db : da) atomicAdd(grad + 12L * body + row, C.gd[q] * u[0]);
            }
            // the four blocks' places, one lane each
            int at = -1;
            if (lane < 4) {
                const int pa = lane >> 1, pb = lane & 1;
                if ((pa ? db : da) && (pb ? db : da)) at = find_block(row_ptr, bcol, pa ? bb : ba, pb ? bb : ba);
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int bi = __shfl_sync(0xffffffffu, at, k);
                if (bi < 0) continue;
                const double (*U)[12] = C.U[k >> 1];
                const double (*Z)[12] = C.Z[k & 1];
                T* V = vals + (long)bi * 144;
                for (int e = lane; e < 144; e += 32) {
                    const int row = e % 12, col = e / 12;          // column-major block entry (row, col)
                    double sum = 0;
#pragma unroll
                    for (int p = 0; p < 5; p++) sum += U[p][row] * Z[p][col];
                    if (sum != 0.0) atomicAdd(V + e, (T)sum);
                }
            }
            __syncwarp();
        }
        __syncwarp();                 // the last types are read before the next contacts' are written
    }
}

// ---------------------------------------------------- block-Jacobi inverse
// One warp per body; a singular block gives the identity.  The Krylov solves'
// preconditioner and the increment of a body that the mixed-precision guard
// replaces; the direct solve inverts the blocks of single bodies itself.
#define BI_WARPS 4
template <class T>
__global__ void __launch_bounds__(32 * BI_WARPS) k_block_inverse(int nb, const int* __restrict__ row_ptr,
        const int* __restrict__ bcol, const T* __restrict__ vals, T* dinv) {
    __shared__ double sM[BI_WARPS][12][25];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double (*M)[25] = sM[w];
    for (int b = blockIdx.x * BI_WARPS + w; b < nb; b += gridDim.x * BI_WARPS) {
        int bi = find_block(row_ptr, bcol, b, b);
        if (bi < 0) continue;
        const bool ok = block_inverse_warp<T>(vals + (long)bi * 144, M, lane);
        T* D = dinv + (long)b * 144;
        for (int e = lane; e < 144; e += 32) {
            int c = e / 12, r = e % 12;
            D[e] = (T)(ok ? M[r][12 + c] : (r == c ? 1.0 : 0.0));
        }
        __syncwarp();
    }
}
int eng_block_inverse(Engine* E) {
    const int nb = E->nb, grid = grid_for(32L * nb, 32 * BI_WARPS);
    int ph = phase_begin(E, PH_ASM_INV);
    if (E->mixed) k_block_inverse<float><<<grid, 32 * BI_WARPS, 0, E->stream>>>(nb, E->row_ptr, E->bcol, (const float*)E->vals, (float*)E->dinv);
    else k_block_inverse<double><<<grid, 32 * BI_WARPS, 0, E->stream>>>(nb, E->row_ptr, E->bcol, (const double*)E->vals, (double*)E->dinv);
    phase_end(E, ph, 0);
    E->launches++;
    return ABD_OK;
}

// waits for the copy the last assembly queued (counters, block keys, done
// flags), not for the assembly kernels behind it
int eng_asm_wait(Engine* E) {
    if (!E->asm_pending) return ABD_OK;
    E->asm_pending = false;
    E->host_syncs++;
    CUDA_TRY(cudaEventSynchronize(E->ev_asm));
    E->keys_host = E->asm_direct;
    E->nnzb_host = E->hcnt->nkeys;   // may include the sentinel
    return ABD_OK;
}

int eng_sync_counters(Engine* E) {
    int rc = eng_asm_wait(E);
    if (rc) return rc;
    CUDA_TRY(cudaMemcpyAsync(E->hcnt, E->dcnt, sizeof(Counters), cudaMemcpyDeviceToHost, E->stream));
    CUDA_TRY(eng_stream_sync(E));
    return ABD_OK;
}

// the counters that the last kernel queued left in pinned memory
// (k_bit_rows run ahead), or a copy of them
int eng_sync_ahead(Engine* E) {
    if (!(E->keys_ahead && E->row_bits)) return eng_sync_counters(E);
    CUDA_TRY(eng_stream_sync(E));
    return ABD_OK;
}

int eng_grow_blocks(Engine* E, int need);

// the contact assembly with the autotuned launch shape: 2, 4 or 8 warps per
// block, one contact per warp until every scheduler of the GPU has a warp
template <class T>
static void launch_contact_assemble(Engine* E, int n, Geo G, double sc, T* V) {
    const AbdParams& P = E->P;
    cudaStream_t s = E->stream;
    int c = tune_begin(E, TK_CONTACT, 3, 1);
    const int threads = TUNE_CONTACT_THREADS[c], warps = TUNE_CONTACT_PER_BLOCK[c];
    int per = 1;
    while (per < CA_PER && (long)per * NUM_SMS * 4 < n) per *= 2;
    dim3 block(threads), grid(grid_for((long)n, warps * per));
#define CA_ARGS E->dcnt, E->cst, E->ctype, E->cxb, G, P.barrier, P.dhat, sc, P.hess_mode, per, E->row_ptr, E->bcol, V, E->g
    if (c == 0) k_contact_assemble<T, 2><<<grid, block, 0, s>>>(CA_ARGS);
    else if (c == 2) k_contact_assemble<T, 8><<<grid, block, 0, s>>>(CA_ARGS);
    else k_contact_assemble<T, 4><<<grid, block, 0, s>>>(CA_ARGS);
#undef CA_ARGS
    tune_end(E, TK_CONTACT);
}

// Block keys: the diagonal and one pair per active contact, sorted and made
// unique, and for the direct solver their copy (with the done flags and the
// counters) to pinned host memory, where its component analysis reads them.
// Exact mode runs inside the assembly, sized by the contact count of the
// last sync, and records an event behind the copies (eng_asm_wait).  Ahead
// mode runs right after the next iterate's detection, before the
// end-of-iteration sync that then brings the keys back as well: the new
// count is not on the host yet, so the keys are sized for the current count
// plus a quarter and 256 (sentinels beyond the device count; a detection
// that found more contacts than that discards them, eng_keys_ahead_synced),
// and no event is needed.
static int asm_keys(Engine* E, bool ahead, long long& bound) {
    cudaStream_t s = E->stream;
    const AbdParams& P = E->P;
    Geo G = eng_geo(E);
    const int nb = E->nb;
    int rc;
    const int n_now = E->hcnt->n_total;
    const int n = ahead ? std::min(E->cap, n_now + n_now / 4 + 256) : n_now;
    if (ahead) E->keys_ahead_n = n;
    const int nkeys = nb + 2 * n;
    // room for every block before the count is known: the unique keys are
    // at most the nkeys written and at most every scene's dense pattern,
    // plus the sentinel
    bound = std::min<long long>(nkeys, E->dense_blocks) + 1;
    if (bound > E->blk_cap) { if ((rc = eng_grow_blocks(E, (int)bound))) return rc; }
    const int ls = E->P.linear_solver;
    const bool direct = ls == ABD_SOLVER_AUTO || ls == ABD_SOLVER_DIRECT;
    if (direct) {
        // rows and columns, or keys of two words
        const long long words = E->row_bits ? nb + 1 + bound : 2LL * nkeys;
        if (words > E->h_pattern_cap) {
            if (E->h_pattern) { CUDA_TRY(eng_stream_sync(E)); cudaFreeHost(E->h_pattern); }
            E->h_pattern = nullptr; E->h_pattern_cap = 0;
            const long long cap = words + words / 2 + 2048;
            if (cudaMallocHost(&E->h_pattern, sizeof(int) * cap) != cudaSuccess)
                return E->fail(ABD_ERR_CUDA, "cudaMallocHost block pattern");
            E->h_pattern_cap = cap;
        }
        if (!E->h_done && cudaMallocHost(&E->h_done, sizeof(int) * E->ns) != cudaSuccess) {
            E->h_done = nullptr;
            return E->fail(ABD_ERR_CUDA, "cudaMallocHost done flags");
        }
    }
    E->keys_host = false;
    E->asm_direct = direct;
    const BitRows B{E->row_bits, E->row_words, E->bscene, E->sc_body_begin};
    int* n_active = B.bits ? &E->dcnt->act : &E->dcnt->n_active;
    if (!B.bits) {
        CUDA_TRY(cudaMemsetAsync(n_active, 0, sizeof(int), s));
        k_diag_keys<<<grid_for(nb), 256, 0, s>>>(nb, E->keys);
    }
    k_contact_prepare<<<grid_for(n > 0 ? n : 1, 128), 128, 0, s>>>(E->dcnt, E->contacts, G, P.ee_f32, P.dhat, nb, E->cap, E->cst,
                                                                   E->ctype, E->cxb, E->cbody, E->keys, B, n_active,
                                                                   ahead ? n : 0);
    if (B.bits) {
        int lanes = 1;
        while (lanes < 32 && lanes < B.words) lanes *= 2;
        BitHost H{nullptr, nullptr, nullptr, E->hcnt};
        if (direct) { H.row = E->h_pattern; H.col = E->h_pattern + nb + 1; H.done = E->h_done; }
        cudaLaunchConfig_t cfg = {};
        const int C = (long)nb * B.words < BR_SPLIT ? 1 : BR_CL;
        cfg.gridDim = dim3(C); cfg.blockDim = dim3(1024); cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        CUDA_TRY(cudaLaunchKernelEx(&cfg, k_bit_rows, nb, (int)bound, B, lanes, E->row_ptr, E->bcol, E->dcnt, E->ns,
                                    (const int*)(E->sci + SI_DONE * E->ns), H));
        E->launches += 2;
        if (!ahead) {
            CUDA_TRY(cudaEventRecord(E->ev_asm, s));
            E->asm_pending = true;
        }
        return ABD_OK;
    }
    int bits = 1;
    while (bits < 64 && ((unsigned long long)nb * nb) >> bits) bits++;
    size_t bytes = E->cub_bytes;
    CUDA_TRY(cub::DeviceRadixSort::SortKeys(E->cub_tmp, bytes, E->keys, E->keys_s, nkeys, 0, bits, s));
    bytes = E->cub_bytes;
    int* n_unique = &E->dcnt->nkeys;
    CUDA_TRY(cub::DeviceSelect::Unique(E->cub_tmp, bytes, E->keys_s, E->ukeys, n_unique, nkeys, s));
    E->launches += 4;
    if (direct) {
        CUDA_TRY(cudaMemcpyAsync(E->h_pattern, E->ukeys, sizeof(unsigned long long) * nkeys, cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaMemcpyAsync(E->h_done, E->sci + SI_DONE * E->ns, sizeof(int) * E->ns, cudaMemcpyDeviceToHost, s));
    }
    if (!ahead) {
        CUDA_TRY(cudaMemcpyAsync(E->hcnt, E->dcnt, sizeof(Counters), cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaEventRecord(E->ev_asm, s));
        E->asm_pending = true;
    }
    return ABD_OK;
}

// the next iterate's block keys, queued before the end-of-iteration sync
int eng_assemble_keys_ahead(Engine* E) {
    long long bound = 0;
    int ph = phase_begin(E, PH_ASM_KEYS);
    int rc = asm_keys(E, true, bound);
    phase_end(E, ph, 0);
    if (rc) return rc;
    E->keys_ahead = true;
    E->keys_ahead_bound = bound;
    return ABD_OK;
}

// after the end-of-iteration sync: keys built ahead are on the host unless
// the detection they came from overflowed (then the assembly rebuilds them)
void eng_keys_ahead_synced(Engine* E) {
    if (!E->keys_ahead) return;
    if (E->hcnt->overflow || E->hcnt->n_total > E->keys_ahead_n) { E->keys_ahead = false; return; }
    E->keys_host = E->asm_direct;
    E->nnzb_host = E->hcnt->nkeys;   // may include the sentinel
}

int eng_assemble(Engine* E) {
    cudaStream_t s = E->stream;
    const AbdParams& P = E->P;
    Geo G = eng_geo(E);
    int nb = E->nb;
    int rc;
    // counters were synchronised by the caller after detection
    int n = E->hcnt->n_total;
    long long bound = 0;
    int ph = phase_begin(E, PH_ASM_KEYS);
    if (E->keys_ahead) {
        bound = E->keys_ahead_bound;      // keys, counters and host copies are there already
        E->keys_ahead = false;
    } else if ((rc = asm_keys(E, false, bound))) {
        return rc;
    }
    if (!E->row_bits) {
        // launch bound; the kernel reads the count from the device
        k_block_rows<<<grid_for(bound), 256, 0, s>>>(nb, E->ukeys, &E->dcnt->nkeys, E->row_ptr, E->bcol, E->dcnt);
        E->launches++;
    }
    phase_end(E, ph, 0);
    double sc = P.kappa * P.dt * P.dt;
    const int per = ba_per(nb);
    if (E->mixed) {
        float* V = (float*)E->vals;
        k_body_assemble<float><<<(nb + per - 1) / per, 32 * BA_WARPS, 0, s>>>(nb, per, E->st, E->mass, E->J, P.dt, P.gravity[0], P.gravity[1], P.gravity[2],
                                                               P.k_ortho, P.hess_mode == ABD_HESS_PROJECTED, P.pinned_diag,
                                                               E->row_ptr, E->bcol, V, E->g);
        if (n > 0)
            launch_contact_assemble<float>(E, n, G, sc, V);
    } else {
        double* V = (double*)E->vals;
        int p1 = phase_begin(E, PH_ASM_BODY);
        k_body_assemble<double><<<(nb + per - 1) / per, 32 * BA_WARPS, 0, s>>>(nb, per, E->st, E->mass, E->J, P.dt, P.gravity[0], P.gravity[1], P.gravity[2],
                                                                P.k_ortho, P.hess_mode == ABD_HESS_PROJECTED, P.pinned_diag,
                                                                E->row_ptr, E->bcol, V, E->g);
        phase_end(E, p1, 0);
        int p2 = phase_begin(E, PH_ASM_CONTACT);
        if (n > 0)
            launch_contact_assemble<double>(E, n, G, sc, V);
        if (E->timing && (rc = eng_asm_wait(E))) return rc;    // n_active for the phase's bytes
        // per candidate: type; per active contact: stencil, barrier argument,
        // 4 positions + 4 rest positions, 4 body blocks and the gradient rows
        phase_end(E, p2, 4.0 * n + E->hcnt->n_active * (16.0 + 8.0 + 96.0 + 96.0 + 4 * 1152.0 + 384.0));
    }
    E->launches += 1 + (n > 0);
    return ABD_OK;
}
