// Host check of the parallel evaluation of serial f64 sums
// (zeno_gb300/csrc/zc_chain.h): rows of 32 values reduced to one function
// each, as the kernel does, against plain serial additions, bit for bit.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "zc_chain.h"

static uint64_t bits_of(double x) {
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
}
static double of_bits(uint64_t b) {
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}

// Rows as the kernel walks them: composed left to right in a tree, a row
// whose result reaches the binade's end re-done by f64 additions.
static double by_rows(double acc, const std::vector<double> &v, std::vector<double> *starts, size_t *serial_rows) {
    for (size_t r = 0; r < v.size(); r += 32) {
        starts->push_back(acc);
        uint32_t e;
        uint64_t m;
        zc::chain_split(bits_of(acc), e, m);
        zc::ChainFn f[32];
        for (size_t j = 0; j < 32; j++) {
            bool tie = false;
            const uint64_t k = r + j < v.size() ? zc::chain_inc(bits_of(v[r + j]), e, tie) : 0;
            f[j] = zc::chain_fn(k, tie);
        }
        for (size_t o = 1; o < 32; o *= 2)
            for (size_t j = 0; j < 32; j += 2 * o) f[j] = zc::chain_then(f[j], f[j + o]);
        const uint64_t end = zc::chain_apply(f[0], m);
        const bool any = f[0].a || f[0].b;
        if (end < zc::kChainCross || !any) {
            acc = any ? of_bits(zc::chain_pack(e, end)) : acc;
        } else {
            (*serial_rows)++;
            for (size_t j = r; j < r + 32 && j < v.size(); j++) acc = acc + v[j];
        }
    }
    return acc;
}

static int check(const char *what, double acc0, const std::vector<double> &v) {
    std::vector<double> starts;
    size_t serial = 0;
    const double got = by_rows(acc0, v, &starts, &serial);
    double acc = acc0;
    for (size_t i = 0; i < v.size(); i++) {
        if (i % 32 == 0 && bits_of(starts[i / 32]) != bits_of(acc) && !(std::isnan(acc) && std::isnan(starts[i / 32]))) {
            std::printf("FAIL %s: start of row %zu\n", what, i / 32);
            return 1;
        }
        acc = acc + v[i];
    }
    if (bits_of(got) != bits_of(acc) && !(std::isnan(got) && std::isnan(acc))) {
        std::printf("FAIL %s: %a against %a\n", what, got, acc);
        return 1;
    }
    return 0;
}

int main() {
    std::mt19937_64 g(12345);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    std::normal_distribution<double> N(0.0, 1.0);
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    const double tiny = std::numeric_limits<double>::denorm_min();
    const size_t sizes[] = {1, 2, 31, 32, 33, 64, 1000, 2048, 2049, 65536};
    int bad = 0, cases = 0;
    for (size_t n : sizes) {
        for (int kind = 0; kind < 12; kind++) {
            std::vector<double> v(n);
            for (size_t i = 0; i < n; i++) {
                const float a = (float)(N(g) * 1e-3), b = (float)(N(g) * 1e-3);
                const double c = N(g) * 1e-3, d = N(g) * 1e-3;
                switch (kind) {
                    case 0: v[i] = c * c + d * d; break;                        // f64 amplitudes
                    case 1: v[i] = (double)a * a + (double)b * b; break;        // f32 amplitudes: many ties
                    case 2: v[i] = std::ldexp(1.0, -(int)(g() % 60)); break;    // powers of two: ties and halves
                    case 3: v[i] = (g() % 7) ? 0.0 : c * c; break;              // sparse
                    case 4: v[i] = std::ldexp((double)(g() % 5), -52); break;   // half-ulps of values near one
                    case 5: v[i] = std::ldexp(U(g), -(int)(g() % 1070)); break; // whole exponent range
                    case 6: v[i] = tiny * (double)(g() % 1000); break;          // subnormals
                    case 7: v[i] = i + 1 == n ? 1.0 : 0.0; break;
                    case 8: v[i] = 1.0 / 65536.0; break;                        // uniform state
                    case 9: v[i] = 0.1; break;
                    case 10: v[i] = i == n / 2 ? inf : c * c; break;
                    default: v[i] = i == n / 2 ? nan : (i == n / 3 ? inf : c * c); break;
                }
            }
            for (double acc0 : {0.0, 0.375, 1.0 - 1e-16, 4503599627370496.0}) {
                bad += check("kind", acc0, v);
                cases++;
            }
        }
    }
    if (bad) return 1;
    std::printf("ok chains %d\n", cases);
    return 0;
}
