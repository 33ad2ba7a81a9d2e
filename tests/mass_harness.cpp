// Host check of the sums of squares of the trajectory engine
// (zeno_gb300/csrc/zc_mass.h) against exact sums: one lane's over many
// additions, and whole table entries with the engine's split of a state over
// lanes, beside the same entries by 256 sums of which each thread holds one.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "zc_mass.h"

using Ops = zc::MassF1;
#ifdef __aarch64__
typedef long double Q;  // 128 bits there
#else
typedef __float128 Q;
#endif

struct Sum {
    float h = 0.f, l = 0.f;
    void add(float x, float y, bool pair = false) {
        if (pair) zc::mass_add_pair<Ops>(x, y, h, l);
        else zc::mass_add2<Ops>(x, y, h, l);
    }
    void fold() { zc::mass_fold<Ops>(h, l); }
    zc::MassSum<Ops> sum3() const { return zc::MassSum<Ops>{h, l, 0.f}; }
    double value() const { return (double)h + (double)l; }
};

static double tree(std::vector<double> v) {
    for (size_t o = v.size() / 2; o; o /= 2)
        for (size_t j = 0; j < o; j++) v[j] += v[j + o];
    return v[0];
}

// A row of M amplitudes as a pass of NT threads sums it: a unit of four
// amplitudes per thread, two pairs (one sum each when NT is 64) of two lanes.
static double row_by_lanes(const std::vector<float> &re, const std::vector<float> &im, size_t NT) {
    const size_t S = NT == 64 ? 2 : 1, units = re.size() / 4;
    std::vector<Sum> sums(NT * 4);
    for (size_t u = 0; u < units; u++)
        for (size_t p = 0; p < 2; p++)
            for (size_t lane = 0; lane < 2; lane++) {
                Sum &s = sums[(u % NT) * 4 + (p % S) * 2 + lane];
                s.add(re[4 * u + 2 * p + lane], im[4 * u + 2 * p + lane], NT >= 256);
                if (p + 1 >= 2 / S && (u / NT) % (zc::kMassFold / 4) == zc::kMassFold / 4 - 1) s.fold();
            }
    // a thread's sums and the lanes of a warp, joined (from eight warps on without
    // the third float down to offset 4); warps added in f64
    std::vector<double> warps;
    for (size_t w = 0; w < NT; w += 32) {
        zc::MassSum<Ops> t[32];
        for (size_t j = 0; j < 32; j++) {
            Sum *s = &sums[4 * (w + j)];
            for (size_t i = 0; i < 4; i++) s[i].fold();
            zc::MassSum<Ops> a = s[0].sum3(), b = s[2].sum3();
            if (NT >= 256) {
                zc::mass_join<false>(a, s[1].sum3());
            } else {
                zc::mass_join<true>(a, s[1].sum3());
                zc::mass_join<true>(b, s[3].sum3());
                zc::mass_join<true>(a, b);
            }
            t[j] = a;
        }
        for (size_t o = 16; o; o /= 2)
            for (size_t j = 0; j < o; j++)
                if (NT >= 256 && o >= 4) zc::mass_join<false>(t[j], t[j + o]);
                else zc::mass_join<true>(t[j], t[j + o]);
        warps.push_back((double)((long double)t[0].h + t[0].l + t[0].c));
    }
    return tree(warps);
}

static double row_by_256(const std::vector<float> &re, const std::vector<float> &im) {
    std::vector<Sum> sums(256);
    for (size_t i = 0; i < re.size(); i++) sums[i % 256].add(re[i], im[i]);
    std::vector<double> v;
    for (Sum &s : sums) v.push_back(s.value());
    return tree(v);
}

int main() {
    std::mt19937 g(11);
    std::normal_distribution<float> gauss;
    // one lane: relative error within the roundings of its additions. A
    // square and a residual are exact; of a pair of squares the two sums of
    // residuals and their sum are rounded (at most 2^-48 of the total each; of
    // a joined pair the FMA's error, its sum with the other and theirs), l is
    // (at most kMassFold + 1/2 ulps, 2^-24 of the total each, before), a fold is
    // exact.
    double worst = 0.0;
    for (int kind = 0; kind < 5; kind++)
        for (int lg = 1; lg <= 18; lg++)
            for (int pair = 0; pair < 2; pair++)
                for (int t = 0; t < (lg <= 12 ? 64 : 4); t++) {
                    const size_t n = (size_t)1 << lg;
                    Sum s;
                    Q exact = 0;
                    float two[2] = {0.f, 0.f};
                    for (size_t i = 0; i < n; i++) {
                        float x = gauss(g) / std::sqrt((float)n);
                        if (kind == 1 && i) x *= 1e-4f;                               // one large amplitude, first
                        if (kind == 2) x = std::ldexp(x, -(int)(g() % 20));           // a wide range
                        if (kind == 3) x *= 1e-9f;                                    // a branch of small mass
                        if (kind == 4 && i + 1 < n) x = g() % 8 ? 0.f : x * 1e-3f;    // sparse, the largest last
                        two[i % 2] = x;
                        exact += (Q)x * x;
                        if (i % 2) s.add(two[0], two[1], pair);
                        if (i % zc::kMassFold == zc::kMassFold - 1) s.fold();
                    }
                    s.fold();
                    const double e = std::fabs((double)(((Q)s.h + (Q)s.l - exact) / exact));
                    const double bound = (double)(n / 2) * std::ldexp(3.0 + zc::kMassFold + 0.5, -48);
                    if (!(e <= bound))
                        return std::printf("FAIL kind %d 2^%d: error %.3e, bound %.3e\n", kind, lg, e, bound), 1;
                    worst = std::max(worst, e / bound);
                }
    // table entries: rms errors over T states, each known to 1 / sqrt(2 T)
    // of itself: three times that of their difference, and the result's own
    // last bit, are let pass
    for (int n : {5, 6, 8, 9, 10, 11, 12, 13, 14, 15, 16, 18, 20})
        for (int K = 1; K <= 2; K++) {
            const size_t M = (size_t)1 << (n - K), NT = n <= 10 ? 64 : n <= 12 ? 128 : n == 13 ? 256 : 512;
            if (M < 4) continue;
            const int T = n <= 14 ? 400 : n <= 16 ? 100 : 10;
            double sq = 0.0, sq_old = 0.0;
            for (int t = 0; t < T; t++) {
                std::vector<float> re(M), im(M);
                Q exact = 0;
                const float sc = 1.f / std::sqrt((float)(2 * M)) * (t % 2 ? 1.f : 1e-5f);
                for (size_t i = 0; i < M; i++) {
                    re[i] = gauss(g) * sc;
                    im[i] = gauss(g) * sc;
                    exact += (Q)re[i] * re[i] + (Q)im[i] * im[i];
                }
                const double e = (double)(((Q)row_by_lanes(re, im, NT) - exact) / exact);
                const double e_old = (double)(((Q)row_by_256(re, im) - exact) / exact);
                sq += e * e;
                sq_old += e_old * e_old;
            }
            const double rms = std::sqrt(sq / T), rms_old = std::sqrt(sq_old / T);
            std::printf("%d qubits, %d-qubit op: %.2e (256 sums %.2e)\n", n, K, rms, rms_old);
            if (rms > rms_old * (1.0 + 3.0 / std::sqrt((double)T)) + std::ldexp(1.0, -54))
                return std::printf("FAIL\n"), 1;
        }
    std::printf("ok sums of squares, at most %.2e of the bound\n", worst);
    return 0;
}
