// Host check of the integer f64 product (zeno_gb300/csrc/zc_softmul.h)
// against the hardware's, bit for bit, over its whole domain.
#include <cstdio>
#include <cstring>
#include <random>

#include "zc_softmul.h"

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

int main() {
    std::mt19937_64 g(7);
    const uint64_t mants[] = {0, 1, 2, 3, 0xfffffffffffffull, 0xffffffffffffeull, 0x8000000000000ull, 0x7ffffffffffffull,
                              0x00000ffffffffull, 0x0000100000000ull, 0x5555555555555ull, 0xaaaaaaaaaaaaaull};
    long checked = 0;
    auto check = [&](uint64_t a, uint64_t b) {
        if (!zc::soft_ok(a) || !zc::soft_ok_right(b)) return true;
        checked++;
        const uint64_t want = bits_of(of_bits(a) * of_bits(b)), got = zc::soft_mul(zc::soft_left(a), zc::soft_right(b));
        if (want != got) std::printf("FAIL %a * %a: %016llx against %016llx\n", of_bits(a), of_bits(b),
                                     (unsigned long long)got, (unsigned long long)want);
        return want == got;
    };
    for (uint64_t ea : {0x200ull, 0x201ull, 0x3fdull, 0x3feull, 0x3ffull, 0x400ull, 0x5feull})
        for (uint64_t eb : {0x300ull, 0x3fdull, 0x3ffull, 0x400ull, 0x4feull})
            for (uint64_t ma : mants)
                for (uint64_t mb : mants)
                    for (int sg = 0; sg < 4; sg++)
                        if (!check(((uint64_t)(sg & 1) << 63) | (ea << 52) | ma, ((uint64_t)(sg >> 1) << 63) | (eb << 52) | mb))
                            return 1;
    for (uint64_t z : {(uint64_t)0, (uint64_t)1 << 63})
        for (uint64_t x : {(uint64_t)0, (uint64_t)1 << 63, bits_of(0.3), bits_of(-1e-50), bits_of(1.0)})
            if (!check(z, x) || !check(x, z)) return 1;
    for (long i = 0; i < 20000000; i++) {
        const uint64_t a = (g() & 0x800fffffffffffffull) | ((0x200 + g() % 0x3ff) << 52);
        uint64_t b = (g() & 0x800fffffffffffffull) | ((0x300 + g() % 0x1ff) << 52);
        if (i % 3 == 0) b &= ~((1ull << (g() % 52)) - 1);  // short mantissas: exact ties and short products
        if (!check(a, b)) return 1;
    }
    std::printf("ok products %ld\n", checked);
    return 0;
}
