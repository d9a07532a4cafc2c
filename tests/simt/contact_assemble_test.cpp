// Driver for tests/test_assembly_kernels_cpu.py: the contact assembly
// (k_contact_assemble of colb_b200/csrc/assemble.cu) under the host emulation of
// simt.h.  The shared memory of a warp is made of Checked values, which count
// every pair of accesses by two lanes, one of them a write, with no warp barrier
// between: such a pair is a race whatever the order in which the
// lanes happen to run.  A small grid makes warps take several groups of
// contacts, with inactive ones at the end of a group; the blocks and the gradient must
// be those of a grid with a warp for every contact.  Exit status 0 when no
// race is counted and all agree to 1e-12 of the largest entry.
#include "simt.h"
#include <mutex>
#include <random>
static thread_local long g_epoch;                         // warp barriers this thread has passed
static long g_first_epoch;                                // of this launch
static std::atomic<long> g_races{0};
static std::mutex g_checked_mu;
template <class T> struct Checked {
    T v;
    mutable long we = -1, re = -1;                        // epochs of the last write and reads
    mutable int wl = -1;
    mutable uint32_t readers = 0;
    operator T() const {
        std::lock_guard<std::mutex> lk(g_checked_mu);
        const int l = threadIdx.x % 32;
        if (we == g_epoch && wl != l) g_races++;
        if (re != g_epoch) { re = g_epoch; readers = 0; }
        readers |= 1u << l;
        return v;
    }
    Checked& operator=(T x) {
        std::lock_guard<std::mutex> lk(g_checked_mu);
        const int l = threadIdx.x % 32;
        if ((we == g_epoch && wl != l) || (re == g_epoch && (readers & ~(1u << l)))) g_races++;
        we = g_epoch; wl = l; v = x;
        return *this;
    }
};
inline void counted_syncwarp() { __syncwarp(); g_epoch++; }
inline int counted_shfl(unsigned m, int v, int src) { const int r = __shfl_sync(m, v, src); g_epoch++; return r; }
#define __syncwarp counted_syncwarp
#define __shfl_sync counted_shfl
#define __shared__ static
#define ABD_HESS_PROJECTED 1
#define ABD_BARRIER_CUBIC 0
#define ABD_BARRIER_QUADRATIC 1
#define T_PP 0
#define T_PE 1
#define T_EE 2
#define T_PT 3
#define T_PG 4
struct int4 { int x, y, z, w; };
struct Counters { int n_total; };
struct Geo { const double* x; const int* vbody; const double* planes; const double* mass; const double* xbar; };
using std::fabs; using std::sqrt; using std::fmax; using std::log; using std::fma;
inline double atomicAdd(double* p, double v) { return std::atomic_ref<double>(*p).fetch_add(v); }
#include "contact_assemble.inc"  // written by the test

int main() {
    const int nb = 3, per_body = 20, n = 75;
    std::mt19937 rng(5);
    std::normal_distribution<double> nd(0.0, 1.0);
    std::vector<double> x(3 * nb * per_body), xbar(x.size()), mass = {1.0, 2.0, 0.0}, planes = {0, 1, 0, -3};
    std::vector<int> vbody(nb * per_body);
    for (auto& v : x) v = nd(rng);
    for (auto& v : xbar) v = nd(rng);
    for (int v = 0; v < nb * per_body; v++) vbody[v] = v / per_body;
    std::vector<int4> cst(n);
    std::vector<int> ctype(n);
    std::vector<double> cxb(n);
    auto vert = [&](int b) { return b * per_body + (int)(rng() % (per_body - 3)); };
    for (int c = 0; c < n; c++) {
        const int a = rng() % nb, b = (a + 1 + rng() % (nb - 1)) % nb, i = vert(a), j = vert(b);
        // inactive: the end of every group of 2, 4 and 8, and some others
        ctype[c] = c % 8 == 7 || c % 4 == 3 || c % 2 == 1 ? -1 : (int)(rng() % 5);
        if (c % 16 == 13) ctype[c] = T_EE;
        cxb[c] = 0.01 + 0.2 * (rng() % 4);
        switch (ctype[c]) {
            case T_PP: cst[c] = {i, j, -1, -1}; break;
            case T_PE: cst[c] = {i, j, j + 1, -1}; break;
            case T_EE: cst[c] = {i, i + 1, j, j + 1}; break;
            case T_PT: cst[c] = {i, j, j + 1, j + 2}; break;
            default: cst[c] = {i, 0, -1, -1};
        }
    }
    Counters cnt{n};
    Geo G{x.data(), vbody.data(), planes.data(), mass.data(), xbar.data()};
    std::vector<int> rp = {0, 3, 6, 9}, col = {0, 1, 2, 0, 1, 2, 0, 1, 2};
    int bad = 0;
    for (int mode = 0; mode < 2; mode++) {
        std::vector<double> ref;
        for (int per : {1, 1, 2, 4, 8}) {
            std::vector<double> out(9 * 144 + 12 * nb, 0.0);
            const bool wide = ref.empty();                // a warp for every contact; after that one block of two warps
            g_first_epoch += 1000000;
            g_races = 0;
            launch(wide ? (n + 1) / 2 : 1, 64, 0, [&] {
                g_epoch = g_first_epoch + 10000L * blockIdx.x;
                k_contact_assemble<double, 2>(&cnt, cst.data(), ctype.data(), cxb.data(), G, 2, 1.0, 3.0, mode, per,
                                              rp.data(), col.data(), out.data(), out.data() + 9 * 144);
            });
            if (wide) ref = out;
            double worst = 0, scale = 0;
            for (size_t i = 0; i < out.size(); i++) {
                worst = std::max(worst, std::fabs(out[i] - ref[i]));
                scale = std::max(scale, std::fabs(ref[i]));
            }
            const bool ok = g_races == 0 && scale > 0 && worst <= 1e-12 * scale;
            printf("mode %d per %d: races %ld, difference %.2e of the largest entry: %s\n", mode, per, g_races.load(),
                   worst / scale, ok ? "ok" : "WRONG");
            bad += !ok;
        }
    }
    return bad;
}
