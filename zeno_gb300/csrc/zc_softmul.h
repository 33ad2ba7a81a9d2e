// The f64 product on the integer pipe, correctly rounded.
//
// GB300's FP64 pipe takes one warp instruction per ~19 cycles per SM, and an
// exact gate is mostly products (16 products and 12 sums per amplitude pair).
// A product of two 53-bit mantissas is four 32 x 32 -> 64 multiplies and about
// twenty integer operations, which issue at several warp instructions per
// cycle, so the products go there and the FP64 pipe keeps the sums.
//
// Valid for operands that are zero or normal with exponents that keep the
// product normal (soft_ok); callers take the FP64 pipe for anything else. The
// rounding is IEEE round-to-nearest-even, the result the same bits.
//
// Compiled for the device (zc_arith.cuh) and for the host
// (tests/softmul_harness.cpp).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define ZC_SM_HD __host__ __device__ __forceinline__
#else
#define ZC_SM_HD inline
#endif

namespace zc {

// One operand, taken apart: the mantissa with its hidden bit, placed so that
// the product of a left and a right operand has 53 or 54 bits above bit 64.
struct SoftOp {
    uint32_t h, l;     // mantissa (left operands << 1, right operands << 11); 0 for zero
    uint32_t e;        // biased exponent (right operands less 1024)
    uint32_t sign;     // bit 31
};

// Zero, or normal with exponent in 2^-511 .. 2^511; the product of two stays
// normal when one of them also passes soft_ok_right (2^-255 .. 2^255).
ZC_SM_HD bool soft_ok(uint64_t b) {
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
    return e - 0x200u < 0x3ffu || (b << 1) == 0;
}
ZC_SM_HD bool soft_ok_right(uint64_t b) {
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
    return e - 0x300u < 0x1ffu || (b << 1) == 0;
}
ZC_SM_HD bool soft_zero(uint64_t b) { return (b << 1) == 0; }

ZC_SM_HD SoftOp soft_left(uint64_t b) {
    const uint32_t hw = (uint32_t)(b >> 32), lw = (uint32_t)b;
    const uint32_t e = (hw >> 20) & 0x7ffu, mh = e ? (hw & 0xfffffu) | 0x100000u : 0u;
    return SoftOp{(mh << 1) | (lw >> 31), lw << 1, e, hw & 0x80000000u};
}
ZC_SM_HD SoftOp soft_right(uint64_t b) {
    const uint32_t hw = (uint32_t)(b >> 32), lw = (uint32_t)b;
    const uint32_t e = (hw >> 20) & 0x7ffu, mh = e ? (hw & 0xfffffu) | 0x100000u : 0u;
    return SoftOp{(mh << 11) | (lw >> 21), lw << 11, e - 1024u, hw & 0x80000000u};
}

ZC_SM_HD uint32_t soft_funnel(uint32_t lo, uint32_t hi, uint32_t s) {  // high word of (hi:lo) << s, s < 32
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

// RN(a * b) as a bit pattern.
ZC_SM_HD uint64_t soft_mul(const SoftOp &a, const SoftOp &b) {
    // 128-bit product, from the bottom: p0.lo, t2.lo, hi (64 bits)
    const uint64_t p0 = (uint64_t)a.l * b.l;
    const uint64_t t1 = (uint64_t)a.l * b.h + (p0 >> 32);
    const uint64_t t2 = (uint64_t)a.h * b.l + (uint32_t)t1;
    const uint64_t hi = (uint64_t)a.h * b.h + (t1 >> 32) + (t2 >> 32);
    const uint32_t h1 = (uint32_t)(hi >> 32), h0 = (uint32_t)hi, r1 = (uint32_t)t2, r0 = (uint32_t)p0;
    // normalise to 54 bits: mantissa and guard
    const uint32_t n = h1 >> 21, s = 1u - n;
    const uint32_t m1 = soft_funnel(h0, h1, s), m0 = soft_funnel(r1, h0, s);
    const uint32_t rest = (soft_funnel(r0, r1, s)) | (r0 << s);
    // round to nearest even: bump by sticky-or-odd, then drop the guard
    const uint32_t bump = (rest ? 1u : 0u) | ((m0 >> 1) & 1u);
    const uint64_t m = ((((uint64_t)m1 << 32) | m0) + bump) >> 1;
    const uint32_t mh = (uint32_t)(m >> 32), ml = (uint32_t)m;
    // the hidden bit adds one to the exponent field (a mantissa rounded up to 2^53 two)
    const uint32_t top = (h1 | h0) ? ((a.e + b.e + n) << 20) + mh : 0u;
    return ((uint64_t)(top | (a.sign ^ b.sign)) << 32) | ml;
}

}  // namespace zc
