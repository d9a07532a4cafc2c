// Driver for tests/test_band_kernel_wide_cpu.py: the band kernel's wide
// instance (body bandwidths 9 to 11) and its signed one (pivots of either sign)
// on diagonally dominant symmetric block-band matrices, each solved as one
// component under the host emulation of simt.h.  The residual of every solution
// must be within 1e-12 of the right-hand side (both in the maximum norm); exit status 0 then.
#include "simt.h"
#include "band_kernel.inc"
#include <random>
template <int BW, bool SIGNED>
static double solve(int N, int wb, int seed) {
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    const int n = 12 * N;
    std::vector<double> M((size_t)n * n, 0.0), g(n);
    for (auto& v : g) v = nd(rng);
    for (int i = 0; i < n; i++)
        for (int j = 0; j < i; j++)
            if (i / 12 - j / 12 <= wb) M[(size_t)i * n + j] = M[(size_t)j * n + i] = 0.3 * nd(rng);
    for (int i = 0; i < n; i++) {
        double s = 1.0;
        for (int j = 0; j < n; j++) s += std::fabs(M[(size_t)i * n + j]);
        M[(size_t)i * n + i] = SIGNED && rng() % 3 == 0 ? -s : s;
    }
    std::vector<int> cptr(1, 0), order, cbw, jobs;
    std::vector<long long> loff;
    long long ltot = 0;
    auto add = [&](int first, int count, int step) {
        loff.push_back(ltot);
        ltot += (long long)count * BW;
        for (int i = 0; i < count; i++) order.push_back(first + i * step);
        cptr.push_back((int)order.size());
        cbw.push_back(wb);
        return (int)cbw.size() - 1;
    };
    const int m = band_split_point(N, wb);
    if (m > 0) {
        const int ct = add(0, m + wb, 1), cb = add(N - 1, N - m, -1);
        jobs = {ct, cb, m};
    } else jobs = {add(0, N, 1), -1, N};
    std::vector<double> Ab((size_t)ltot * 144, 0.0), Lg((size_t)ltot * 144 + 12 * order.size(), 0.0), du(n, 0.0);
    for (size_t c = 0; c + 1 < cptr.size(); c++)
        for (int i = 0; i < cptr[c + 1] - cptr[c]; i++)
            for (int d = 0; d <= std::min(wb, i); d++) {
                const int bi = order[cptr[c] + i], bj = order[cptr[c] + i - d];
                for (int e = 0; e < 144; e++)
                    Ab[((size_t)loff[c] + (size_t)i * BW + d) * 144 + e] = M[(size_t)(12 * bi + e / 12) * n + 12 * bj + e % 12];
            }
    int status = 0;
    launch(2, BAND_THREADS, (size_t)band_smem_doubles(BW) * 8, [&] {
        k_band_solve<BW, SIGNED>(1, jobs.data(), cptr.data(), order.data(), cbw.data(), loff.data(), Ab.data(), ltot,
                                 g.data(), Lg.data(), du.data(), &status);
    }, 2);
    double worst = 0, scale = 0;
    for (int i = 0; i < n; i++) {
        double r = -g[i];
        for (int j = 0; j < n; j++) r += M[(size_t)i * n + j] * du[j];
        worst = std::max(worst, std::fabs(r)); scale = std::max(scale, std::fabs(g[i]));
    }
    printf("N %d wb %d signed %d: residual %.3e status %d\n", N, wb, (int)SIGNED, worst / scale, status);
    return status == 0 && worst <= 1e-12 * scale ? 0 : 1;
}
int main() {
    int bad = 0;
    bad += solve<BAND_WIDE + 1, false>(10, 9, 1) + solve<BAND_WIDE + 1, false>(29, 9, 2);
    bad += solve<BAND_WIDE + 1, false>(32, 10, 3) + solve<BAND_WIDE + 1, false>(12, 11, 4);
    bad += solve<BAND_WIDE + 1, true>(35, 11, 5) + solve<BAND_WIDE + 1, true>(20, 9, 6);
    bad += solve<BAND_W, true>(3, 1, 7) + solve<BAND_W, true>(24, 5, 8) + solve<BAND_W, true>(28, 8, 9);
    return bad;
}
