// Sums of squares in two floats.
//
// (h, l) holds a sum as h + l. A square y^2 = p + e is split exactly (one
// product, one FMA), p joins h by TwoSum (Knuth), whose error is exact whatever
// the sizes, and both errors go to l. The sum starts at zero, so its error is
// relative to the sum itself: a branch of small mass keeps its digits. l is a
// plain sum of errors; it is folded back into h every kMassFold squares, or
// with their number its own roundings would come to show.
// Shorter forms are less exact: the residual of an FMA h + y^2 is rounded once
// more, always down a little (the low bits of a square are not uniform), and a
// sum on top of a constant keeps digits of the constant, not of the sum.
// Relative error of a table entry over a 16-qubit state (Gaussian amplitudes):
// 1e-15 by these sums, 4e-15 with the FMA residual, 1.3e-12 on top of 1.
//
// Written over Ops (one float, or two packed in a register pair); compiled for
// the device (zc_traj.cu) and for the host (tests/mass_harness.cpp).
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define ZC_MASS_HD __host__ __device__ __forceinline__
#else
#define ZC_MASS_HD inline
#endif

namespace zc {

constexpr int kMassFold = 64;  // squares between two folds

// The operations on one float.
struct MassF1 {
    typedef float V;
    static ZC_MASS_HD float zero() { return 0.f; }
    static ZC_MASS_HD float neg(float a) { return -a; }
    static ZC_MASS_HD void by_size(float x, float y, float &a, float &b) {  // a NaN stays one of the two
        const bool first = fabsf(x) >= fabsf(y);
        a = fabsf(first ? x : y);
        b = fabsf(first ? y : x);
    }
#ifdef __CUDA_ARCH__
    static ZC_MASS_HD float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    static ZC_MASS_HD float add(float a, float b) { return __fadd_rn(a, b); }
    static ZC_MASS_HD float sub(float a, float b) { return __fsub_rn(a, b); }
#else
    static ZC_MASS_HD float fma(float a, float b, float c) { return ::fmaf(a, b, c); }
    static ZC_MASS_HD float add(float a, float b) { return a + b; }
    static ZC_MASS_HD float sub(float a, float b) { return a - b; }
#endif
};

// h += p; returns TwoSum's error.
template <typename Ops>
ZC_MASS_HD typename Ops::V mass_two_sum(typename Ops::V &h, typename Ops::V p) {
    const typename Ops::V s = Ops::add(h, p), b = Ops::sub(s, h);
    const typename Ops::V e = Ops::add(Ops::sub(h, Ops::sub(s, b)), Ops::sub(p, b));
    h = s;
    return e;
}

// (h, l) += x^2 + y^2.
template <typename Ops>
ZC_MASS_HD void mass_add2(typename Ops::V x, typename Ops::V y, typename Ops::V &h, typename Ops::V &l) {
    const typename Ops::V o = Ops::zero();
    // the squares as FMAs: a product that feeds a sum may be contracted with it
    const typename Ops::V p = Ops::fma(x, x, o), q = Ops::fma(y, y, o);
    const typename Ops::V ep = Ops::fma(x, x, Ops::neg(p)), eq = Ops::fma(y, y, Ops::neg(q));
    const typename Ops::V rp = mass_two_sum<Ops>(h, p), rq = mass_two_sum<Ops>(h, q);
    l = Ops::add(l, Ops::add(Ops::add(rp, rq), Ops::add(ep, eq)));
}

// The same in 14 operations instead of 20, with two more roundings, each of the
// last bit of x^2 + y^2: the larger square's product takes the other by an FMA,
// whose error is one more FMA because their difference is exact (Sterbenz:
// p <= s <= 2p), and only that sum joins h. For CTAs whose sums are many (NT >=
// 256), where the roundings average out: 118 -> 113 ms for 2048 trajectories at
// 16 qubits.
template <typename Ops>
ZC_MASS_HD void mass_add_pair(typename Ops::V x, typename Ops::V y, typename Ops::V &h, typename Ops::V &l) {
    typename Ops::V a, b;
    Ops::by_size(x, y, a, b);  // |a| >= |b|
    const typename Ops::V p = Ops::fma(a, a, Ops::zero()), ep = Ops::fma(a, a, Ops::neg(p));
    const typename Ops::V s = Ops::fma(b, b, p);
    const typename Ops::V e = Ops::add(Ops::fma(b, b, Ops::sub(p, s)), ep);
    const typename Ops::V r = mass_two_sum<Ops>(h, s);
    l = Ops::add(l, Ops::add(r, e));
}

// The same sum with |l| at most half an ulp of h.
template <typename Ops>
ZC_MASS_HD void mass_fold(typename Ops::V &h, typename Ops::V &l) {
    const typename Ops::V s = Ops::add(h, l);
    l = Ops::sub(l, Ops::sub(s, h));
    h = s;
}

// A folded sum on its way through the additions over lanes.
template <typename Ops>
struct MassSum {
    typename Ops::V h, l, c;
};

// a += b. THIRD: c takes what h and l lose, so that the sum keeps ~2^-70 and a
// table of few values is as good as they are. Without it 2^-48, for the
// additions of many values, whose roundings average out.
template <bool THIRD, typename Ops>
ZC_MASS_HD void mass_join(MassSum<Ops> &a, const MassSum<Ops> &b) {
    typename Ops::V s = a.h, t = a.l;
    const typename Ops::V e = mass_two_sum<Ops>(s, b.h);
    if (THIRD) {
        const typename Ops::V f = mass_two_sum<Ops>(t, b.l), g = mass_two_sum<Ops>(t, e);
        a.c = Ops::add(Ops::add(a.c, b.c), Ops::add(f, g));
    } else {
        t = Ops::add(e, Ops::add(t, b.l));
    }
    a.h = Ops::add(s, t);
    a.l = Ops::sub(t, Ops::sub(a.h, s));
}

}  // namespace zc
