// Serial f64 sums of non-negative values, evaluated in parallel, bit for bit.
//
// A chain acc = RN(acc + v_0), RN(acc + v_1), ... looks serial: every rounding
// depends on the sum before it. But while acc stays in one binade its ulp is
// fixed, acc = M * 2^e with M an integer below 2^53, and adding v moves M by
// v / 2^e rounded to the nearest integer, whatever M is. Only an exact tie
// looks at M, and only at its parity (ties go to the even M). So each v is a
// function of M's parity, M -> M + (M even ? a : b), such functions compose
// associatively, and a run of elements reduces to one of them: integer adds
// in any tree order. The one element whose sum leaves the binade (M reaches
// 2^53), and elements larger than the binade, are added as f64 instead;
// a chain over 2^16 values crosses about sixteen binades.
//
// Compiled for the device (zc_reduce.cu) and for the host
// (tests/chain_harness.cpp).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define ZC_HD __host__ __device__ __forceinline__
#else
#define ZC_HD inline
#endif

namespace zc {

constexpr uint64_t kChainCross = 1ull << 53;  // M at the end of the binade; also "larger than the binade"

// A non-negative f64 bit pattern as m * 2^(e - 1075), e >= 1 (zero and
// subnormals share e = 1 with the smallest normal binade).
ZC_HD void chain_split(uint64_t bits, uint32_t &e, uint64_t &m) {
    const uint32_t f = (uint32_t)(bits >> 52);
    e = f ? f : 1u;
    m = (bits & 0xfffffffffffffull) | (f ? 1ull << 52 : 0ull);
}

// The bit pattern of m * 2^(e - 1075) for m <= 2^53 (m below 2^52 only where e = 1).
ZC_HD uint64_t chain_pack(uint32_t e, uint64_t m) { return ((uint64_t)(e - 1) << 52) + m; }

// M -> M + (M even ? a : b).
struct ChainFn {
    uint64_t a, b;
};

// f, then g.
ZC_HD ChainFn chain_then(const ChainFn &f, const ChainFn &g) {
    return ChainFn{f.a + ((f.a & 1) ? g.b : g.a), f.b + ((f.b & 1) ? g.a : g.b)};
}
ZC_HD uint64_t chain_apply(const ChainFn &f, uint64_t m) { return m + ((m & 1) ? f.b : f.a); }

// What adding the value of `vbits` does to M in the binade e: k, or on a tie
// (k even with M, else k + 1). Values beyond the binade (and inf, NaN) give
// kChainCross; with the accumulator inf or NaN (e = 0x7ff) every value does.
ZC_HD uint64_t chain_inc(uint64_t vbits, uint32_t e, bool &tie) {
    uint32_t ev;
    uint64_t mv;
    chain_split(vbits, ev, mv);
    tie = false;
    if (e == 0x7ffu) return kChainCross;
    if (ev >= e) return ev == e ? mv : kChainCross;
    const uint32_t d = e - ev;
    if (d > 53) return 0;
    const uint64_t rem = mv & ((1ull << d) - 1), half = 1ull << (d - 1);
    tie = rem == half;
    return (mv >> d) + (rem > half);
}
ZC_HD ChainFn chain_fn(uint64_t k, bool tie) {
    return tie ? ChainFn{k + (k & 1), k + 1 - (k & 1)} : ChainFn{k, k};
}

}  // namespace zc
