// Driver for tests/test_assembly_kernels_cpu.py: the block rows' pattern from
// bits (k_bit_rows of colb_b200/csrc/assemble.cu) under the host emulation of
// simt.h, by one block and by a cluster.  A store into another block's
// shared memory is only allowed once the storing thread has waited for a
// cluster barrier, that is, once every block of the cluster is known to run;
// one that comes earlier is counted and not carried out.  Exit status 0 when
// there is none and rows, columns and counters are those of the bits.
#include "simt.h"
#include <random>
static int g_cluster;                                     // blocks of the cluster
static std::vector<unsigned char*> g_base(8);             // their shared memory
static std::atomic<int> g_early{0};
static thread_local int g_phases;                         // cluster barriers this thread has passed
inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
inline int __shfl_up_sync(unsigned m, int v, int o, int = 32) {
    const int l = threadIdx.x % 32;
    return (int)__shfl_sync(m, (double)v, l >= o ? l - o : l);
}
inline int __shfl_sync(unsigned m, int v, int src, int) { return (int)__shfl_sync(m, (double)v, src); }
inline uint32_t br_cluster_blocks() { return g_cluster; }
inline uint32_t br_cluster_rank() { return blockIdx.x % g_cluster; }
inline void br_cluster_arrive() { band_cluster_arrive(); }
inline void br_cluster_wait() { band_cluster_wait(); g_phases++; }
inline void br_store(int* p, int rank, int v) {
    if (g_phases == 0) { g_early++; return; }
    *reinterpret_cast<int*>(g_base[rank] + (reinterpret_cast<unsigned char*>(p) - g_dyn_smem)) = v;
}
struct Counters { int nnzb, nkeys, n_active, act; };
#include "bit_rows.inc"  // written by the test

static int run(int nb, int cluster, int per_row, int seed) {
    const int words = (nb + 31) / 32;                     // one scene; from 17 words on a warp reads a row
    std::mt19937 rng(seed);
    std::vector<uint32_t> bits((size_t)nb * words, 0);
    std::vector<std::vector<char>> on(nb, std::vector<char>(nb, 0));
    for (int k = 0; k < nb * per_row / 2; k++) {
        const int a = rng() % nb, b = rng() % nb;
        if (a == b) continue;
        on[a][b] = on[b][a] = 1;
        bits[(size_t)a * words + b / 32] |= 1u << (b % 32);
        bits[(size_t)b * words + a / 32] |= 1u << (a % 32);
    }
    std::vector<int> rp(1, 0), col;
    for (int r = 0; r < nb; r++) {
        for (int c = 0; c < nb; c++) if (on[r][c] || r == c) col.push_back(c);
        rp.push_back((int)col.size());
    }
    const int bound = (int)col.size() + 7;
    std::vector<int> row_ptr(nb + 1, -1), bcol(bound, -1), hrow(nb + 1, -1), hcol(bound, -1), bscene(nb, 0), begin = {0, nb};
    int done[1] = {1}, hdone[1] = {0};
    Counters cnt = {0, 0, 0, 42}, hcnt = {0, 0, 0, 0};
    BitRows B{bits.data(), words, bscene.data(), begin.data()};
    BitHost H{hrow.data(), hcol.data(), hdone, &hcnt};
    g_cluster = cluster;
    launch(cluster, 1024, 4096, [&] {
        g_base[blockIdx.x] = g_dyn_smem;
        g_phases = 0;
        k_bit_rows(nb, bound, B, 32, row_ptr.data(), bcol.data(), &cnt, 1, done, H);
    }, cluster);
    bcol.resize(col.size());
    hcol.resize(col.size());
    bool ok = row_ptr == rp && bcol == col && hrow == rp && hcol == col && hdone[0] == 1 && cnt.nnzb == rp[nb] &&
              cnt.nkeys == rp[nb] && cnt.n_active == 42 && cnt.act == 0 && hcnt.nnzb == rp[nb] && hcnt.n_active == 42;
    for (uint32_t w : bits) ok = ok && w == 0;
    printf("bodies %d cluster %d: blocks %d, early stores %d: %s\n", nb, cluster, rp[nb], g_early.load(), ok ? "ok" : "WRONG");
    return ok && g_early == 0 ? 0 : 1;
}
int main() {
    return run(520, 1, 3, 1) + run(520, 2, 3, 2) + run(1030, 2, 6, 3) + run(545, 3, 0, 4);
}
