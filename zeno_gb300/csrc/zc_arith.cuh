// Arithmetic policy for the gate kernels.
//
// EXACT = true reproduces zeno's scalar CPU kernels bit for bit: every
// product and sum is a separately rounded IEEE operation (the __*_rn
// intrinsics are never contracted into FMA), evaluated in the reference's
// left-to-right order (src/state.rs:253-256, :382-383, :521-525, :592-593).
// EXACT = false lets the update use fused multiply-adds (tolerance parity).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "zc_softmul.h"

namespace zc {

template <typename T>
struct Vec;
template <>
struct Vec<double> {
    using type = double2;  // 16-byte vector access
    static constexpr int N = 2;
};
template <>
struct Vec<float> {
    using type = float4;
    static constexpr int N = 4;
};

__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

template <typename T>
struct Mat2 {
    T v[8];  // m00r m00i m01r m01i m10r m10i m11r m11i
};

// Exact f64 arithmetic with the products on the integer pipe (zc_softmul.h)
// and the sums on the FP64 pipe. Operands outside the integer product's domain
// (subnormals, inf, NaN, extreme exponents) take the FP64 pipe for everything.
__device__ __forceinline__ uint64_t f64_bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double soft_product(const SoftOp &a, const SoftOp &b) {
    return __longlong_as_double((long long)soft_mul(a, b));
}

// A 2x2 matrix (m00r m00i m01r m01i m10r m10i m11r m11i) for exact updates:
// which entries are nonzero, and whether all are in the product's domain with
// a nonzero entry in each row.
struct ExactMask {
    uint32_t nz;  // bit i: entry i nonzero
    bool soft;
};
__device__ __forceinline__ ExactMask exact_mask(const double *m) {
    ExactMask k{0, true};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint64_t b = f64_bits(m[i]);
        k.nz |= soft_zero(b) ? 0u : 1u << i;
        k.soft &= soft_ok_right(b);
    }
    k.soft &= (k.nz & 0x0fu) && (k.nz & 0xf0u);
    return k;
}

// The reference's update of the pair (a, b), bit for bit: each row is
// ((m0 * ar - m1 * ai) + m2 * br) - m3 * bi and its imaginary twin. A term of
// a zero entry is exactly +-0 and leaves a sum as it is unless the sum is a
// zero too; with four nonzero inputs no partial sum is a negative zero, so
// such terms are left out (a u3 gate has one, H and RY four, RX four).
// The FP64 pipe bounds it: 28 -> 12 operations per pair (10 for a u3).
// Measured over 96 u3 gates and 48 CX at 24 qubits: 44.6 -> 26.0 ms, the FP64
// pipe still busy 74% of the time.
__device__ __forceinline__ void pair_update_f64(const double *m, const ExactMask &k, double &ar, double &ai, double &br,
                                                double &bi) {
    const uint64_t b0 = f64_bits(ar), b1 = f64_bits(ai), b2 = f64_bits(br), b3 = f64_bits(bi);
    if (k.soft && soft_ok(b0) && soft_ok(b1) && soft_ok(b2) && soft_ok(b3)) {
        const bool zero = soft_zero(b0) || soft_zero(b1) || soft_zero(b2) || soft_zero(b3);
        const uint32_t nz = zero ? 0xffu : k.nz;
        const SoftOp xar = soft_left(b0), xai = soft_left(b1), xbr = soft_left(b2), xbi = soft_left(b3);
        double re[2], im[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            double x = 0.0, y = 0.0;
            if (nz & (1u << (4 * r))) {
                const SoftOp w = soft_right(f64_bits(m[4 * r]));
                x = soft_product(xar, w);
                y = soft_product(xai, w);
            }
            if (nz & (2u << (4 * r))) {
                const SoftOp w = soft_right(f64_bits(m[4 * r + 1]));
                x = rsub(x, soft_product(xai, w));
                y = radd(y, soft_product(xar, w));
            }
            if (nz & (4u << (4 * r))) {
                const SoftOp w = soft_right(f64_bits(m[4 * r + 2]));
                x = radd(x, soft_product(xbr, w));
                y = radd(y, soft_product(xbi, w));
            }
            if (nz & (8u << (4 * r))) {
                const SoftOp w = soft_right(f64_bits(m[4 * r + 3]));
                x = rsub(x, soft_product(xbi, w));
                y = radd(y, soft_product(xbr, w));
            }
            re[r] = x;
            im[r] = y;
        }
        ar = re[0];
        ai = im[0];
        br = re[1];
        bi = im[1];
        return;
    }
    const double nar = rsub(radd(rsub(rmul(m[0], ar), rmul(m[1], ai)), rmul(m[2], br)), rmul(m[3], bi));
    const double nai = radd(radd(radd(rmul(m[0], ai), rmul(m[1], ar)), rmul(m[2], bi)), rmul(m[3], br));
    const double nbr = rsub(radd(rsub(rmul(m[4], ar), rmul(m[5], ai)), rmul(m[6], br)), rmul(m[7], bi));
    const double nbi = radd(radd(radd(rmul(m[4], ai), rmul(m[5], ar)), rmul(m[6], bi)), rmul(m[7], br));
    ar = nar;
    ai = nai;
    br = nbr;
    bi = nbi;
}

// One exact f64 product a * w (w in the right operand's domain or not).
__device__ __forceinline__ bool soft_pair_ok(double a, double b, double w, double v) {
    return soft_ok(f64_bits(a)) && soft_ok(f64_bits(b)) && soft_ok_right(f64_bits(w)) && soft_ok_right(f64_bits(v));
}

// 2x2 complex update of the pair (a, b) = (bit q clear, bit q set)
// (kern_1q_scalar, src/state.rs:251-257).
template <typename T, bool EXACT>
__device__ __forceinline__ void pair_update(const Mat2<T> &m, T &ar, T &ai, T &br, T &bi) {
    const T m00r = m.v[0], m00i = m.v[1], m01r = m.v[2], m01i = m.v[3];
    const T m10r = m.v[4], m10i = m.v[5], m11r = m.v[6], m11i = m.v[7];
    T nar, nai, nbr, nbi;
    if constexpr (EXACT) {
        nar = rsub(radd(rsub(rmul(m00r, ar), rmul(m00i, ai)), rmul(m01r, br)), rmul(m01i, bi));
        nai = radd(radd(radd(rmul(m00r, ai), rmul(m00i, ar)), rmul(m01r, bi)), rmul(m01i, br));
        nbr = rsub(radd(rsub(rmul(m10r, ar), rmul(m10i, ai)), rmul(m11r, br)), rmul(m11i, bi));
        nbi = radd(radd(radd(rmul(m10r, ai), rmul(m10i, ar)), rmul(m11r, bi)), rmul(m11i, br));
    } else {
        nar = rfma(-m01i, bi, rfma(m01r, br, rfma(-m00i, ai, m00r * ar)));
        nai = rfma(m01i, br, rfma(m01r, bi, rfma(m00i, ar, m00r * ai)));
        nbr = rfma(-m11i, bi, rfma(m11r, br, rfma(-m10i, ai, m10r * ar)));
        nbi = rfma(m11i, br, rfma(m11r, bi, rfma(m10i, ar, m10r * ai)));
    }
    ar = nar;
    ai = nai;
    br = nbr;
    bi = nbi;
}

// Complex scale of one amplitude by (wr, wi) (kern_diag*_scalar,
// src/state.rs:521-525, :592-593): re' = wr*ar - wi*ai, im' = wr*ai + wi*ar.
template <typename T, bool EXACT>
__device__ __forceinline__ void cscale(T wr, T wi, T &ar, T &ai) {
    T nr, ni;
    if constexpr (EXACT && sizeof(T) == 8) {
        if (soft_pair_ok(ar, ai, wr, wi)) {  // products on the integer pipe
            const SoftOp xr = soft_left(f64_bits(ar)), xi = soft_left(f64_bits(ai));
            const SoftOp vr = soft_right(f64_bits(wr)), vi = soft_right(f64_bits(wi));
            nr = rsub(soft_product(xr, vr), soft_product(xi, vi));
            ni = radd(soft_product(xi, vr), soft_product(xr, vi));
        } else {
            nr = rsub(rmul(wr, ar), rmul(wi, ai));
            ni = radd(rmul(wr, ai), rmul(wi, ar));
        }
    } else if constexpr (EXACT) {
        nr = rsub(rmul(wr, ar), rmul(wi, ai));
        ni = radd(rmul(wr, ai), rmul(wi, ar));
    } else {
        nr = rfma(-wi, ai, wr * ar);
        ni = rfma(wi, ar, wr * ai);
    }
    ar = nr;
    ai = ni;
}

// One term of the fused k-qubit matvec (kern_kq_scalar, src/state.rs:382-383):
// ar = (ar + wr*xr) - wi*xi ; ai = (ai + wr*xi) + wi*xr.
// SOFT: exact f64 products on the integer pipe, for callers with enough of them
// in flight. (k_kq's rows, one product after another from shared memory, took
// longer with it: 7 qubits on 12 623 -> 681 us, on 24 33.3 -> 33.6 ms.)
template <typename T, bool EXACT, bool SOFT = false>
__device__ __forceinline__ void cmac(T wr, T wi, T xr, T xi, T &ar, T &ai) {
    if constexpr (EXACT && SOFT && sizeof(T) == 8) {
        double p0, p1, p2, p3;
        if (soft_pair_ok(xr, xi, wr, wi)) {  // products on the integer pipe
            const SoftOp sr = soft_left(f64_bits(xr)), si = soft_left(f64_bits(xi));
            const SoftOp vr = soft_right(f64_bits(wr)), vi = soft_right(f64_bits(wi));
            p0 = soft_product(sr, vr);
            p1 = soft_product(si, vi);
            p2 = soft_product(si, vr);
            p3 = soft_product(sr, vi);
        } else {
            p0 = rmul(wr, xr);
            p1 = rmul(wi, xi);
            p2 = rmul(wr, xi);
            p3 = rmul(wi, xr);
        }
        ar = rsub(radd(ar, p0), p1);
        ai = radd(radd(ai, p2), p3);
    } else if constexpr (EXACT) {
        ar = rsub(radd(ar, rmul(wr, xr)), rmul(wi, xi));
        ai = radd(radd(ai, rmul(wr, xi)), rmul(wi, xr));
    } else {
        ar = rfma(-wi, xi, rfma(wr, xr, ar));
        ai = rfma(wi, xr, rfma(wr, xi, ai));
    }
}

// ------------------------------------------------------------------
// Double-float arithmetic for f64 states (fast mode).
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so the f64 kernels' fast
// mode keeps the state in f64 in HBM but does the gate arithmetic on the
// FP32 pipe with unevaluated (hi, lo) float pairs (Dekker 1971; error-free
// TwoSum of Knuth, two-product via FMA). Conversions between f64 and the
// pair use integer and FP32 operations only, never the FP64 pipe. A general
// gate costs about 43 FP32 operations per output component and carries
// ~2^-46 relative error; f64 -> pair and pair -> f64 round to nearest (2^-48 and
// 2^-53 of hi). Zero, subnormals and |x| < 2^-126 map to 0.

// f64 -> (hi, lo): hi = x truncated to 24 bits, lo the next 23, rounded by the
// 24th (ties away) or, DOWN, truncated. Rounded, a sum over many values keeps no
// bias: truncated ones left P(1) of a 20-qubit state 7e-15 low.
template <bool DOWN = false>
__device__ __forceinline__ float2 df_from_f64(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned hw = (unsigned)(b >> 32), lw = (unsigned)b;
    const int e = (int)((hw >> 20) & 0x7ff);
    const unsigned sign = hw & 0x80000000u;
    const int ef = e - 896;   // f32 exponent field of hi
    const int efl = e - 919;  // exponent placing the low bits below hi
    const unsigned mant23 = ((hw & 0xfffffu) << 3) | (lw >> 29);
    float hi = 0.0f, lo = 0.0f;
    if (ef >= 1 && ef <= 254) hi = __uint_as_float(sign | ((unsigned)ef << 23) | mant23);
    if (efl >= 1 && ef <= 254) {
        const unsigned top = sign | ((unsigned)efl << 23);
        const unsigned up = DOWN ? 0u : (lw >> 5) & 1u;  // carries into the exponent: lo is one ulp of hi then
        lo = __fsub_rn(__uint_as_float((top | ((lw >> 6) & 0x7fffffu)) + up), __uint_as_float(top));
    }
    return make_float2(hi, lo);
}

// Exact f32 -> f64 widening with integer operations only (the FP64 pipe's
// conversion shares its slow issue rate). Subnormals are normalised; inf and
// NaN keep their class.
__device__ __forceinline__ double f32_to_f64_exact(float x) {
    const unsigned u = __float_as_uint(x);
    const unsigned long long sign = (unsigned long long)(u >> 31) << 63;
    const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
    unsigned long long bits;
    if (e == 0xffu) {
        bits = sign | (0x7ffull << 52) | ((unsigned long long)m << 29);
    } else if (e != 0u) {
        bits = sign | ((unsigned long long)(e + 896u) << 52) | ((unsigned long long)m << 29);
    } else if (m == 0u) {
        bits = sign;
    } else {
        const int sh = __clz(m) - 8;  // brings the leading one to bit 23
        bits = sign | ((unsigned long long)(897 - sh) << 52) | ((unsigned long long)((m << sh) & 0x7fffffu) << 29);
    }
    return __longlong_as_double((long long)bits);
}
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) { return f32_to_f64_exact(x); }

// (hi, lo) -> f64 for |lo| <= ulp(hi): the f64 bit pattern of hi plus lo
// counted in f64 ulps of hi's binade (|lo| <= 2^28 of them; one binade lower
// when hi is a power of two and lo points down, where the ulp halves), scaled
// by a power of two and rounded to an integer: the f64 nearest hi + lo.
// |hi| < 2^-75 keeps hi alone; zero and subnormal hi give 0.
__device__ __forceinline__ double df_to_f64(float2 v) {
    const unsigned hb = __float_as_uint(v.x), lb = __float_as_uint(v.y);
    const unsigned eh = (hb >> 23) & 0xffu;
    if (eh == 0u) return 0.0;
    const unsigned mant = hb & 0x7fffffu;
    const unsigned long long hbits =
        ((unsigned long long)((hb & 0x80000000u) | ((eh + 896u) << 20) | (mant >> 3)) << 32) |
        (unsigned long long)(mant << 29);
    const bool down = mant == 0u && ((hb ^ lb) & 0x80000000u) && (lb & 0x7fffffffu);
    const unsigned se = 306u - eh + (down ? 1u : 0u);  // f32 exponent field of 2^(179 - eh (+1))
    if (se >= 255u) return __longlong_as_double((long long)hbits);
    const int L = __float2int_rn(__fmul_rn(v.y, __uint_as_float(se << 23)));
    return __longlong_as_double((long long)(hbits + (unsigned long long)(long long)((hb >> 31) ? -L : L)));
}

// Exact product split: a*b = p + e with e from one FMA, plus cross terms.
__device__ __forceinline__ void df_prod(float2 a, float2 b, float &p, float &e) {
    p = __fmul_rn(a.x, b.x);
    e = __fmaf_rn(a.x, b.x, -p);
    e = __fmaf_rn(a.x, b.y, e);
    e = __fmaf_rn(a.y, b.x, e);
}

// s + err = a + b exactly (TwoSum).
__device__ __forceinline__ float two_sum(float a, float b, float &err) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return s;
}

__device__ __forceinline__ float2 df_norm(float s, float lo) {
    const float h = __fadd_rn(s, lo);
    return make_float2(h, __fsub_rn(lo, __fsub_rn(h, s)));
}

__device__ __forceinline__ float2 df_neg(float2 a) { return make_float2(-a.x, -a.y); }

// x0*y0 + x1*y1 + x2*y2 + x3*y3 in double-float.
__device__ __forceinline__ float2 df_dot4(float2 x0, float2 y0, float2 x1, float2 y1, float2 x2, float2 y2, float2 x3,
                                          float2 y3) {
    float p0, e0, p1, e1, p2, e2, p3, e3, r1, r2, r3;
    df_prod(x0, y0, p0, e0);
    df_prod(x1, y1, p1, e1);
    df_prod(x2, y2, p2, e2);
    df_prod(x3, y3, p3, e3);
    float s = two_sum(p0, p1, r1);
    s = two_sum(s, p2, r2);
    s = two_sum(s, p3, r3);
    const float lo = __fadd_rn(__fadd_rn(__fadd_rn(r1, r2), r3), __fadd_rn(__fadd_rn(e0, e1), __fadd_rn(e2, e3)));
    return df_norm(s, lo);
}

// The residual of a sum with a rounded product p = fl(x y) in it: TwoSum's last
// difference p - pp (pp: p as the sum sees it) plus the product's own rounding
// error x y - p is x y - pp, one FMA, rounded once where the two were added.
// A sum of two products so takes 8 operations for hi and residual (against 13
// for two split products and a TwoSum), x + t y takes 7 (against 9).

// x0*y0 + x1*y1 in double-float, unnormalised.
__device__ __forceinline__ float2 df_dot2_u(float2 x0, float2 y0, float2 x1, float2 y1) {
    const float p0 = __fmul_rn(x0.x, y0.x), p1 = __fmul_rn(x1.x, y1.x);
    const float s = __fadd_rn(p0, p1);
    const float b = __fsub_rn(s, p0), a = __fsub_rn(s, b);
    float l0 = __fmaf_rn(x0.x, y0.x, -a), l1 = __fmaf_rn(x1.x, y1.x, -b);
    l0 = __fmaf_rn(x0.x, y0.y, l0);
    l1 = __fmaf_rn(x1.x, y1.y, l1);
    l0 = __fmaf_rn(x0.y, y0.x, l0);
    l1 = __fmaf_rn(x1.y, y1.x, l1);
    return make_float2(s, __fadd_rn(l0, l1));
}
__device__ __forceinline__ float2 df_dot2(float2 x0, float2 y0, float2 x1, float2 y1) {
    const float2 r = df_dot2_u(x0, y0, x1, y1);
    return df_norm(r.x, r.y);
}

// Gate matrix in double-float: m00r m00i m01r m01i m10r m10i m11r m11i.
struct MatDF {
    float2 v[8];
};

// Host-exact split of the f64 entries happens on the device once per op.
__device__ __forceinline__ MatDF df_matrix(const double *m) {
    MatDF r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = df_from_f64(m[i]);
    return r;
}

// 2x2 complex update of (a, b) in double-float (same formula as pair_update).
__device__ __forceinline__ void pair_update_df(const MatDF &m, float2 &ar, float2 &ai, float2 &br, float2 &bi) {
    const float2 nar = df_dot4(m.v[0], ar, df_neg(m.v[1]), ai, m.v[2], br, df_neg(m.v[3]), bi);
    const float2 nai = df_dot4(m.v[0], ai, m.v[1], ar, m.v[2], bi, m.v[3], br);
    const float2 nbr = df_dot4(m.v[4], ar, df_neg(m.v[5]), ai, m.v[6], br, df_neg(m.v[7]), bi);
    const float2 nbi = df_dot4(m.v[4], ai, m.v[5], ar, m.v[6], bi, m.v[7], br);
    ar = nar;
    ai = nai;
    br = nbr;
    bi = nbi;
}

// Real 2x2 update (r00 r01 r10 r11) of (a, b) in double-float: four
// two-term dot products instead of the complex update's four-term ones.
__device__ __forceinline__ void pair_update_rdf(const float2 *r, float2 &ar, float2 &ai, float2 &br, float2 &bi) {
    const float2 nar = df_dot2(r[0], ar, r[1], br);
    const float2 nai = df_dot2(r[0], ai, r[1], bi);
    const float2 nbr = df_dot2(r[2], ar, r[3], br);
    const float2 nbi = df_dot2(r[2], ai, r[3], bi);
    ar = nar;
    ai = nai;
    br = nbr;
    bi = nbi;
}

// Unnormalised variants (also df_dot2_u above) for chains of operations
// inside one register pass: the (s, lo) pair is left as the sum and its error
// terms give it (|lo| a few ulps of s at most); products and sums of the next
// operation stay exact in their hi parts whatever the pair's normalisation, so
// the chain keeps the double-float error bound relative to its inputs. df_norm
// once at the end.

// x + t*y in double-float.
__device__ __forceinline__ float2 df_axpy_u(float2 x, float2 t, float2 y) {
    const float p = __fmul_rn(t.x, y.x);
    const float s = __fadd_rn(x.x, p);
    const float b = __fsub_rn(s, x.x);
    const float da = __fsub_rn(x.x, __fsub_rn(s, b));
    // the small terms first: x.y may have grown over a chain
    float lo = __fadd_rn(da, __fmaf_rn(t.x, y.x, -b));
    lo = __fmaf_rn(t.x, y.y, lo);
    lo = __fmaf_rn(t.y, y.x, lo);
    return make_float2(s, __fadd_rn(x.y, lo));
}

__device__ __forceinline__ float2 df_renorm(float2 v) { return df_norm(v.x, v.y); }

__device__ __forceinline__ void cscale_df_u(float2 wr, float2 wi, float2 &ar, float2 &ai) {
    const float2 nr = df_dot2_u(wr, ar, df_neg(wi), ai);
    const float2 ni = df_dot2_u(wr, ai, wi, ar);
    ar = nr;
    ai = ni;
}

__device__ __forceinline__ void cscale_df(float2 wr, float2 wi, float2 &ar, float2 &ai) {
    const float2 nr = df_dot2(wr, ar, df_neg(wi), ai);
    const float2 ni = df_dot2(wr, ai, wi, ar);
    ar = nr;
    ai = ni;
}

// ------------------------------------------------------------------
// Packed double-float arithmetic (f32x2).
//
// add / sub / mul / fma .rn.f32x2 apply one IEEE FP32 operation to both
// halves of a 64-bit register pair. The FP32 datapath does the same number
// of operations per clock either way, but a packed instruction takes one
// issue slot and one step of a dependency chain for two of them. The
// double-float sweeps therefore hold a complex amplitude as
//   H = (re hi, im hi),  L = (re lo, im lo)
// and run the real and imaginary halves of a rotation through one
// instruction stream. Each half sees the operations of the scalar
// routines above in the same order; where a routine subtracts a value, the
// packed one may add its negative (negation is exact and rounding to nearest
// is symmetric), so both give the same values (a zero may carry the other
// sign).

__device__ __forceinline__ unsigned long long pk_bits(float2 v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ float2 pk_float2(unsigned long long r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pk_bits(a)), "l"(pk_bits(b)));
    return pk_float2(d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pk_bits(a)), "l"(pk_bits(b)));
    return pk_float2(d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pk_bits(a)), "l"(pk_bits(b)), "l"(pk_bits(c)));
    return pk_float2(d);
}

// A real double-float coefficient t as pairs: (t hi, t hi), (t lo, t lo) and
// their negatives.
struct PkReal {
    float2 h, l, nh, nl;
};

// x + t*y per half: df_axpy_u on (H, L) pairs (h, l the pairs of t).
__device__ __forceinline__ void pk_axpy_u(float2 h, float2 l, float2 Hx, float2 Lx, float2 Hy, float2 Ly, float2 &Hr,
                                          float2 &Lr) {
    // the product as an FMA: a packed mul whose only use is an add gets
    // contracted with it (measured: results lose the low parts)
    const float2 s = add2(Hx, fma2(h, Hy, make_float2(0.f, 0.f)));
    const float2 nb = sub2(Hx, s);
    const float2 da = sub2(Hx, add2(s, nb));
    float2 lo = add2(da, fma2(h, Hy, nb));
    lo = fma2(h, Ly, lo);
    lo = fma2(l, Hy, lo);
    Hr = s;
    Lr = add2(Lx, lo);
}

// [[1, -t], [t, 1]] on (a, b), unnormalised.
__device__ __forceinline__ void pk_rot_u(const PkReal &t, float2 &Ha, float2 &La, float2 &Hb, float2 &Lb) {
    float2 Hn, Ln;
    pk_axpy_u(t.nh, t.nl, Ha, La, Hb, Lb, Hn, Ln);
    pk_axpy_u(t.h, t.l, Hb, Lb, Ha, La, Hb, Lb);
    Ha = Hn;
    La = Ln;
}

// (H, L) <-> the scalar routines' (re, im) double-float pairs.
__device__ __forceinline__ void pk_split(float2 H, float2 L, float2 &ar, float2 &ai) {
    ar = make_float2(H.x, L.x);
    ai = make_float2(H.y, L.y);
}
__device__ __forceinline__ void pk_join(float2 ar, float2 ai, float2 &H, float2 &L) {
    H = make_float2(ar.x, ai.x);
    L = make_float2(ar.y, ai.y);
}

// Renormalise both halves (df_norm per half).
__device__ __forceinline__ void pk_renorm(float2 &H, float2 &L) {
    const float2 h = add2(H, L);
    L = sub2(L, sub2(h, H));
    H = h;
}

// f64 (re, im) <-> packed pairs; to_f64 renormalises first.
__device__ __forceinline__ void pk_from_f64(double re, double im, float2 &H, float2 &L) {
    pk_join(df_from_f64(re), df_from_f64(im), H, L);
}
__device__ __forceinline__ void pk_to_f64(float2 H, float2 L, double &re, double &im) {
    pk_renorm(H, L);
    re = df_to_f64(make_float2(H.x, L.x));
    im = df_to_f64(make_float2(H.y, L.y));
}

// Arithmetic policies: 0 = exact reference trees, 1 = FMA-contracted,
// 2 = double-float on the FP32 pipe (f64 states only).
enum : int { AR_EXACT = 0, AR_FMA = 1, AR_DF = 2 };

// pair_update under policy A on values stored as T.
template <typename T, int A>
__device__ __forceinline__ void upd2(const Mat2<T> &m, const MatDF &md, T &ar, T &ai, T &br, T &bi) {
    if constexpr (A == AR_DF) {
        float2 xr = df_from_f64(ar), xi = df_from_f64(ai), yr = df_from_f64(br), yi = df_from_f64(bi);
        pair_update_df(md, xr, xi, yr, yi);
        ar = df_to_f64(xr);
        ai = df_to_f64(xi);
        br = df_to_f64(yr);
        bi = df_to_f64(yi);
    } else if constexpr (A == AR_EXACT && sizeof(T) == 8) {
        pair_update_f64(m.v, exact_mask(m.v), ar, ai, br, bi);  // the mask is loop-invariant in every caller
    } else {
        pair_update<T, A == AR_EXACT>(m, ar, ai, br, bi);
    }
}

template <typename T, int A>
__device__ __forceinline__ void scale2(T wr, T wi, float2 wrd, float2 wid, T &ar, T &ai) {
    if constexpr (A == AR_DF) {
        float2 xr = df_from_f64(ar), xi = df_from_f64(ai);
        cscale_df(wrd, wid, xr, xi);
        ar = df_to_f64(xr);
        ai = df_to_f64(xi);
    } else {
        cscale<T, A == AR_EXACT>(wr, wi, ar, ai);
    }
}

// insert_zeros (src/state.rs:162-169): spread g around zero bits at the
// ascending positions qs[0..k).
__device__ __forceinline__ uint64_t insert_zeros(uint64_t g, const uint32_t *qs, int k) {
    uint64_t x = g;
    for (int i = 0; i < k; i++) {
        const uint32_t q = qs[i];
        const uint64_t low = x & ((1ull << q) - 1);
        x = ((x >> q) << (q + 1)) | low;
    }
    return x;
}

__device__ __forceinline__ uint64_t insert_zero(uint64_t h, uint32_t q) {
    return ((h >> q) << (q + 1)) | (h & ((1ull << q) - 1));
}

}  // namespace zc
