// Driver for tests/test_band_check_cpu.py: the signed band kernel on symmetric
// block-band matrices that are indefinite and not diagonally dominant, some
// with a leading pivot of zero or near it, and the check of its solution
// (band_check), both from colb_b200/csrc/dense.cu under the host emulation of simt.h.
// The entries are FP32 values.  A solution whose largest row-wise backward
// error, in long double, is above four times the check's bound must be
// marked, one below a quarter of it must not be, and the matrices say which they are.
#include "simt.h"
#include <cfloat>
#include "band_kernel.inc"
#include "band_check.inc"
constexpr int WARPS = 4;
static void check_all(int nb, const int* rp, const int* col, const float* vals, const double* g, const double* du, int* bad) {
    static int transposed[WARPS][32];
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    for (int b = w; b < nb; b += WARPS) band_check<float>(b, nb, lane, transposed[w], rp, col, vals, g, du, bad);
}
#include <random>
enum Kind { DOMINANT, INDEFINITE, TINY_PIVOT, ZERO_PIVOT, NOT_FINITE };
template <int BW>
static int run(int N, int wb, Kind kind, double pivot, int seed) {
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    const int n = 12 * N;
    std::vector<double> M((size_t)n * n, 0.0), g(n);
    for (auto& v : g) v = nd(rng);
    for (int i = 0; i < n; i++)
        for (int j = 0; j <= i; j++)
            if (i / 12 - j / 12 <= wb) M[(size_t)i * n + j] = M[(size_t)j * n + i] = (double)(float)nd(rng);
    for (int i = 0; i < n; i++) {
        double s = 1.0;
        for (int j = 0; j < n; j++) s += std::fabs(M[(size_t)i * n + j]);
        if (kind == DOMINANT) M[(size_t)i * n + i] = (double)(float)(i % 3 ? s : -s);
        else M[(size_t)i * n + i] = (double)(float)((i % 2 ? 4.0 : -4.0) * std::sqrt(12.0 * wb));   // below the row's sum
    }
    if (kind == TINY_PIVOT || kind == ZERO_PIVOT) M[0] = (double)(float)pivot;
    if (kind == NOT_FINITE) M[0] = INFINITY;
    std::vector<int> cptr = {0, N}, order, cbw = {wb}, jobs = {0, -1, N};
    std::vector<long long> loff = {0};
    for (int i = 0; i < N; i++) order.push_back(i);
    const long long ltot = (long long)N * BW;
    std::vector<double> Ab((size_t)ltot * 144, 0.0), Lg((size_t)ltot * 144 + 12 * N, 0.0), du(n, 0.0);
    std::vector<int> rp = {0}, col;
    std::vector<float> vals;
    for (int i = 0; i < N; i++) {
        for (int j = std::max(0, i - wb); j <= std::min(N - 1, i + wb); j++) {
            col.push_back(j);
            for (int e = 0; e < 144; e++) vals.push_back((float)M[(size_t)(12 * i + e % 12) * n + 12 * j + e / 12]);
        }
        rp.push_back((int)col.size());
        for (int d = 0; d <= std::min(wb, i); d++)
            for (int e = 0; e < 144; e++)
                Ab[((size_t)i * BW + d) * 144 + e] = M[(size_t)(12 * i + e / 12) * n + 12 * (i - d) + e % 12];
    }
    int status = 0;
    launch(2, BAND_THREADS, (size_t)band_smem_doubles(BW) * 8, [&] {
        k_band_solve<BW, true>(1, jobs.data(), cptr.data(), order.data(), cbw.data(), loff.data(), Ab.data(), ltot,
                               g.data(), Lg.data(), du.data(), &status);
    }, 2);
    std::vector<int> bad(N + 1, 0);
    launch(1, 32 * WARPS, 0, [&] { check_all(N, rp.data(), col.data(), vals.data(), g.data(), du.data(), bad.data()); });
    long double worst = 0;
    for (int i = 0; i < n; i++) {
        long double r = g[i], s = std::fabs(g[i]);
        for (int j = 0; j < n; j++) { r -= (long double)M[(size_t)i * n + j] * du[j]; s += std::fabs((long double)M[(size_t)i * n + j] * du[j]); }
        const long double e = std::fabs(r) / s;
        if (worst == worst && !(e <= worst)) worst = e;       // a NaN stays
    }
    bool ok = true;
    if (!(worst <= 4 * BAND_BACKWARD)) ok = ok && bad[N];
    if (worst < BAND_BACKWARD / 4) ok = ok && !bad[N];
    if (kind == DOMINANT) ok = ok && !bad[N];
    if (kind == ZERO_PIVOT || kind == TINY_PIVOT || kind == NOT_FINITE) ok = ok && bad[N];
    bool any = false;
    for (int b = 0; b < N; b++) any = any || bad[b];
    ok = ok && any == (bad[N] != 0);
    printf("bodies %d bandwidth %d kind %d pivot %g: backward error %.2Le, %s: %s\n", N, wb, (int)kind, pivot, worst,
           bad[N] ? "marked" : "kept", ok ? "ok" : "WRONG");
    return !ok;
}
int main() {
    int bad = 0;
    bad += run<BAND_W>(3, 1, DOMINANT, 0, 1) + run<BAND_W>(7, 5, DOMINANT, 0, 2) + run<BAND_WIDE + 1>(14, 11, DOMINANT, 0, 3);
    for (int seed = 10; seed < 13; seed++) bad += run<BAND_W>(9, 4, INDEFINITE, 0, seed) + run<BAND_WIDE + 1>(12, 9, INDEFINITE, 0, seed);
    for (double p : {1e-13, -1e-15, 1e-30}) bad += run<BAND_W>(6, 3, TINY_PIVOT, p, 20) + run<BAND_WIDE + 1>(12, 10, TINY_PIVOT, p, 21);
    bad += run<BAND_W>(2, 1, ZERO_PIVOT, 0, 30) + run<BAND_W>(10, 8, ZERO_PIVOT, 0, 31) + run<BAND_WIDE + 1>(12, 11, ZERO_PIVOT, 0, 32);
    bad += run<BAND_W>(4, 2, NOT_FINITE, 0, 40);
    return bad;
}
