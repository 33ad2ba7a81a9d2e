// Batched noisy trajectories: every trajectory of a noisy run in ONE launch.
//
// zeno runs a noisy circuit one shot at a time (src/exec.rs:459-549): each
// shot replays the ops and, after every gate, the channels of
// src/noise.rs:145-175 — depolarizing, then per touched qubit bit flip,
// phase flip and amplitude damping (whose jump probability gamma * P(1)
// needs a reduction over the state), then readout flips at measurement.
//
// Here a persistent CTA owns one trajectory at a time. Per op the CTA makes
// one pass over the state that (a) applies the previous op's pending noise
// operators that are diagonal as a per-element factor, (b) applies the gate
// (times the depolarizing Pauli string drawn for this op), and (c) accumulates
// the joint probability table of the op's qubits. Warp 0 then resolves flips
// and damping for the touched qubits in the reference's order on that table
// (each decision updates the table), leaves the resulting 2x2 operators
// pending for the next pass and prepares the next op; two CTA barriers per op.
// All draws of an op are independent of the state and come in the
// reference's order from a per-trajectory Philox4x32-10 stream
// (zc_philox.h). Probabilities are summed in two floats per lane and three over
// lanes (zc_mass.h), and over warps in FP64.
//
// Where the state lives. The pass is bound by moving the state (2S per op),
// so it stays as close as it fits: up to 14 qubits (128 KiB) in shared
// memory; above, the first part in shared memory and the rest in a per-CTA
// buffer, one CTA per SM so that all SMs' buffers stay in the L2 (16 qubits:
// 152 x 320 KiB = 47 MiB).
//
// The pass moves 16-byte vectors and works on four independent groups per
// thread (the vector's lanes) as packed f32x2 arithmetic; ops on qubits 0 and
// 1 permute lanes in registers (see lanes). While a gate's pass runs, warp 1
// prepares the next op (look_ahead), so that only what the table decides
// stands between two passes. Measured for 2048 trajectories of the 16-qubit
// depth-20 circuit under damping: 402 ms with one scalar pass per op over
// global memory (114 instructions per amplitude, four CTAs per SM, half the
// traffic from DRAM), 113 ms now (16 us per op and SM; bound by the latency of
// the L2 half of the state, the sums of squares and the decisions between
// passes; 106 with sums on top of a constant, which lost digits of small ones,
// see zc_mass.h); 1500 shots of a 13-qubit dynamic circuit: 10.2 -> 2.2 ms.
// Measured and dropped: two units
// per thread for one-qubit ops (+17%, registers), 256-bit accesses to an
// interleaved global part (2x, spills), passes out of line (+20%).
#include <algorithm>

#include "zc_arith.cuh"
#include "zc_internal.h"
#include "zc_mass.h"
#include "zc_philox.h"
#include "zc_traj.h"

namespace zc {
namespace {

// ---------------------------------------------------------------- complex helpers

// Complex values of the per-op operators (gate x Pauli string, pending noise
// operators, diagonal factors): single precision, like the f32 states they act
// on (GB300's FP64 pipe would make thread 0's serial work the bottleneck);
// branch probabilities stay FP64.
struct C2 {
    float re, im;
};
__device__ __forceinline__ C2 cmul(C2 a, C2 b) { return C2{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return C2{a.re + b.re, a.im + b.im}; }

// Pauli by code 1 = X, 2 = Y, 3 = Z as a 2x2 row-major complex matrix.
__device__ void pauli(int code, C2 *m) {
    for (int i = 0; i < 4; i++) m[i] = C2{0, 0};
    if (code == 1) m[1] = m[2] = C2{1, 0};
    if (code == 2) m[1] = C2{0, -1}, m[2] = C2{0, 1};
    if (code == 3) m[0] = C2{1, 0}, m[3] = C2{-1, 0};
    if (code == 0) m[0] = m[3] = C2{1, 0};
}

// out = a . b for 2x2.
__device__ void mul22(const C2 *a, const C2 *b, C2 *out) {
    C2 r[4];
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++) r[i * 2 + j] = cadd(cmul(a[i * 2], b[j]), cmul(a[i * 2 + 1], b[2 + j]));
    for (int i = 0; i < 4; i++) out[i] = r[i];
}

struct Pending {
    uint32_t q;
    C2 m[4];
};

// Ring of Philox blocks held ahead: at least 32 when a pass begins, of which
// its op takes at most nine (three per qubit) and the next one two.
constexpr uint32_t kDraws = 64;

template <int NT>
struct Shared {
    float4 w[2][64];              // op matrix (gate x Pauli string): (re, re, im, im) per entry
    float2 nw[2][64];             // (-im, -im)
    float4 ft[8];                 // diagonal pending factor per vector lane, by the high factor bits
    TrajRec recs[4];              // op i's record at i % 4: the pass's, the next, the one being copied in
    int o;                        // behind finish_op: the op of the next pass (nops at the end),
    int cur;                      //   whose matrix is w[cur]
    uint32_t xm[2];               // row flips of the op's Pauli string
    int look[2];                  // by o % 2: how far look_ahead got with op o + 1 (LOOK_*)
    int look_draws;               // draws that took
    Pending pend[3];              // operators left by the previous op's noise that are not diagonal
    int npend;                    //   (three-qubit ops: all of them, until their tables are built)
    uint32_t fqv[3];              // high qubits of the factor table, in vector units
    int nfv;                      // -1: no factor differs from one
    uint32_t dq[3];               // all qubits of the diagonal factors, and the factors by their bits
    float dr[8];
    int nd;
    double red[NT / 32][8];       // per-warp tables
    double J[8];                  // joint probability table of a three-qubit op
    double seg[32], blk[32];      // final sampling: region and block masses
    double el[1024];              //   and the element masses of one block
    double us[kDraws];            // draw i at i % kDraws: as f64, and the integer half of the block
    uint64_t zw[kDraws];
    uint64_t draw, drawn;         // stream positions of the next draw and behind the last one held
    double keep, keep2;           // sqrt(1 - gamma), 1 - gamma
    uint64_t cl;                  // classical bits of this trajectory
    double u;                     // final sampling: what is left of the draw
    int region, block;
    __device__ __forceinline__ const TrajOp &op(int i) const { return recs[i & 3].op; }
};

// The next op is still to be found (LOOK_NO); its matrix is ready (LOOK_READY);
// ready, and this op leaves nothing to decide either (LOOK_GO).
enum : int { LOOK_NO = 0, LOOK_READY = 1, LOOK_GO = 2 };

// An op's probability table is read: measurements, and gates under damping.
__device__ __forceinline__ bool wants_table(const TrajOp &op, const TrajNoise &nz) {
    return op.kind != TOP_GATE || nz.on(4);
}

// The CTA's tables. Functions reach them here rather than by reference, so
// that those kept out of line still address shared memory directly.
template <int NT>
__device__ __forceinline__ Shared<NT> &shared_of() {
    __shared__ Shared<NT> s;
    return s;
}

// Two f32 lanes in one 64-bit register pair, the form loads, stores and the
// packed arithmetic share.
typedef unsigned long long P2;
__device__ __forceinline__ P2 p2_make(float x, float y) { return pk_bits(make_float2(x, y)); }
__device__ __forceinline__ P2 p2_mul(P2 a, P2 b) {
    P2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ P2 p2_fma(P2 a, P2 b, P2 c) {
    P2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ P2 p2_add(P2 a, P2 b) {
    P2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ P2 p2_sub(P2 a, P2 b) {
    P2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Where the trajectory's state is: amplitudes below ns in shared memory, the
// others in the CTA's global buffer. SMEM: all of it in shared memory.
template <bool SMEM>
struct StateMem {
    float *sre, *sim, *gre, *gim;
    uint64_t ns;
    // work: the CTA's global buffer (2^(n + 1) floats), unused if SMEM
    __device__ __forceinline__ StateMem(float *work, uint32_t n) {
        extern __shared__ __align__(16) float smem[];
        ns = 1ull << n;
        if (!SMEM && ns > kTrajSplitElems) ns = kTrajSplitElems;
        sre = smem;
        sim = smem + ns;
        gre = work;
        gim = work + (1ull << n);
    }
    __device__ __forceinline__ float &re(uint64_t i) const { return SMEM || i < ns ? sre[i] : gre[i]; }
    __device__ __forceinline__ float &im(uint64_t i) const { return SMEM || i < ns ? sim[i] : gim[i]; }
    // vector v (amplitudes 4v .. 4v + 3) as two pairs
    __device__ __forceinline__ ulonglong2 *re4(uint32_t v) const {
        return reinterpret_cast<ulonglong2 *>(SMEM || v < (uint32_t)(ns >> 2) ? sre : gre) + v;
    }
    __device__ __forceinline__ ulonglong2 *im4(uint32_t v) const {
        return reinterpret_cast<ulonglong2 *>(SMEM || v < (uint32_t)(ns >> 2) ? sim : gim) + v;
    }
};

// Apply every non-diagonal pending operator as a 1-qubit pass.
template <int NT, bool SMEM>
__device__ __noinline__ void apply_nondiag_pending(float *work, uint32_t n) {
    Shared<NT> &s = shared_of<NT>();
    const StateMem<SMEM> sm(work, n);
    const uint64_t half = 1ull << (n - 1);
    for (int p = 0; p < s.npend; p++) {
        const Pending &P = s.pend[p];
        const float m00r = P.m[0].re, m00i = P.m[0].im, m01r = P.m[1].re, m01i = P.m[1].im;
        const float m10r = P.m[2].re, m10i = P.m[2].im, m11r = P.m[3].re, m11i = P.m[3].im;
        for (uint64_t h = threadIdx.x; h < half; h += NT) {
            const uint64_t a = insert_zero(h, P.q), b = a | (1ull << P.q);
            const float ar = sm.re(a), ai = sm.im(a), br = sm.re(b), bi = sm.im(b);
            sm.re(a) = m00r * ar - m00i * ai + m01r * br - m01i * bi;
            sm.im(a) = m00r * ai + m00i * ar + m01r * bi + m01i * br;
            sm.re(b) = m10r * ar - m10i * ai + m11r * br - m11i * bi;
            sm.im(b) = m10r * ai + m10i * ar + m11r * bi + m11i * br;
        }
        __syncthreads();
    }
}

// Per-element factor of the diagonal pending operators.
template <int NT>
__device__ __forceinline__ float diag_factor(const Shared<NT> &s, uint64_t idx) {
    uint32_t j = 0;
    for (int b = 0; b < s.nd; b++) j |= (uint32_t)((idx >> s.dq[b]) & 1) << b;
    return s.dr[j];
}

// Warp 0, every lane with the same arguments: the tables of the real diagonal
// factors (f0[b], f1[b]) on qubits q[b], b < nd, per element and per vector.
template <int NT>
__device__ __forceinline__ void factor_tables(Shared<NT> &s, int nd, const uint32_t *q, const float *f0,
                                              const float *f1) {
    const int lane = threadIdx.x % 32;
    bool one = true;
    int nfv = 0;
    float f = 1.f, fv = 1.f;  // this lane's entry per element (bits: lane), per vector (lane & 3, lane >> 2)
#pragma unroll
    for (int b = 0; b < 3; b++)
        if (b < nd) {
            one &= f0[b] == 1.f && f1[b] == 1.f;
            f = __fmul_rn(f, (lane >> b) & 1 ? f1[b] : f0[b]);
            const int bit = q[b] < 2 ? (lane >> q[b]) & 1 : (lane >> (2 + nfv)) & 1;
            fv = __fmul_rn(fv, bit ? f1[b] : f0[b]);
            if (q[b] >= 2) {
                if (lane == 0) s.fqv[nfv] = q[b] - 2;
                nfv++;
            }
            if (lane == 0) s.dq[b] = q[b];
        }
    if (lane < 8) s.dr[lane] = f;
    reinterpret_cast<float *>(s.ft)[lane] = fv;
    if (lane == 0) {
        s.nd = nd;
        s.nfv = one ? -1 : nfv;
    }
}

// The same from the pending list of a three-qubit op, which also keeps only
// its operators that are not diagonal. (All operators are real.)
template <int NT>
__device__ void split_pending(Shared<NT> &s) {
    uint32_t q[3] = {0, 0, 0};
    float f0[3] = {1.f, 1.f, 1.f}, f1[3] = {1.f, 1.f, 1.f};
    int nd = 0, np = 0;
    for (int p = 0; p < s.npend; p++) {
        const Pending P = s.pend[p];
        if (P.m[1].re == 0 && P.m[2].re == 0) {
            q[nd] = P.q;
            f0[nd] = P.m[0].re;
            f1[nd++] = P.m[3].re;
        } else {
            __syncwarp();
            if (threadIdx.x == 0) s.pend[np] = P;
            np++;
        }
    }
    factor_tables(s, nd, q, f0, f1);
    __syncwarp();
    if (threadIdx.x == 0) s.npend = np;
}

// The operations of zc_mass.h on two lanes.
struct MassF2 {
    typedef P2 V;
    static __device__ __forceinline__ P2 zero() { return 0ull; }
    static __device__ __forceinline__ P2 fma(P2 a, P2 b, P2 c) { return p2_fma(a, b, c); }
    static __device__ __forceinline__ P2 add(P2 a, P2 b) { return p2_add(a, b); }
    static __device__ __forceinline__ P2 sub(P2 a, P2 b) { return p2_sub(a, b); }
    static __device__ __forceinline__ P2 neg(P2 a) { return a ^ 0x8000000080000000ull; }
    static __device__ __forceinline__ void by_size(P2 x, P2 y, P2 &a, P2 &b) {
        const float2 u = pk_float2(x), v = pk_float2(y);
        a = p2_make(larger(u.x, v.x), larger(u.y, v.y));
        b = p2_make(smaller(u.x, v.x), smaller(u.y, v.y));
    }
    // of two magnitudes, NaN if either is
    static __device__ __forceinline__ float larger(float x, float y) {
        float r;
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(fabsf(x)), "f"(fabsf(y)));
        return r;
    }
    static __device__ __forceinline__ float smaller(float x, float y) {
        float r;
        asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(fabsf(x)), "f"(fabsf(y)));
        return r;
    }
};

// Table values on their way through a warp: float sums (zc_mass.h), not FP64, of
// which an SM takes one warp instruction per 19 cycles (9 qubits, 2048
// trajectories: 1.70 ms with FP64 additions, 1.20 so). CTAs of eight warps and
// more have many values and join them without the third float down to the
// lowest four lanes (2048 trajectories at 16 qubits: 114 -> 112 ms).
typedef MassSum<MassF1> Sum3;

// The f64 nearest h + l + c, by integer operations: as df_to_f64, with c and what
// rounding l to f64 units left added in those units. Masses are scaled by 2^48
// on the way, below 2^-123 they are h alone.
__device__ __forceinline__ double mass_f64(const Sum3 &v) {
    const float h = v.h * 0x1p48f, t = v.l + v.c, l = t * 0x1p48f, c = (v.c - (t - v.l)) * 0x1p48f;
    const unsigned hb = __float_as_uint(h), eh = hb >> 23, mant = hb & 0x7fffffu;  // h >= 0
    if (eh == 0u) return 0.0;
    if (eh == 255u) return (double)v.h;  // inf, NaN
    const long long hbits = (long long)((unsigned long long)((eh + 896u - 48u) << 20 | mant >> 3) << 32 |
                                        (unsigned long long)(mant << 29));
    const unsigned se = 306u - eh + (mant == 0u && l < 0.f ? 1u : 0u);  // f32 exponent field of 1 / (f64 unit)
    if (se >= 255u) return __longlong_as_double(hbits);
    const float units = __uint_as_float(se << 23), f = __fmul_rn(l, units);
    const int L = __float2int_rn(f);
    return __longlong_as_double(hbits + L + __float2int_rn(__fmaf_rn(c, units, __fsub_rn(f, (float)L))));
}

template <bool THIRD>
__device__ __forceinline__ Sum3 sum_of(Sum3 a, const Sum3 &b) {
    mass_join<THIRD>(a, b);
    return a;
}
// Both lanes of a sum.
template <bool THIRD>
__device__ __forceinline__ Sum3 mass_end(P2 h, P2 l) {
    mass_fold<MassF2>(h, l);
    const float2 a = pk_float2(h), b = pk_float2(l);
    return sum_of<THIRD>(Sum3{a.x, b.x, 0.f}, Sum3{a.y, b.y, 0.f});
}
__device__ __forceinline__ Sum3 shfl_xor_of(const Sum3 &v, int m) {
    return Sum3{__shfl_xor_sync(0xffffffffu, v.h, m), __shfl_xor_sync(0xffffffffu, v.l, m),
                __shfl_xor_sync(0xffffffffu, v.c, m)};
}

// The warp's table into red[0..D) from D sums per thread: lanes halve the values
// they carry as they exchange them (D - 1 + 5 - log2 D additions instead of 5 D).
template <int D, int NT>
__device__ __forceinline__ void warp_table(Sum3 *v, double *red) {
    constexpr bool THIRD = NT < 256;
    const int lane = threadIdx.x % 32;
    int off = 16, base = 0;
#pragma unroll
    for (int w = D; w > 1; w >>= 1, off >>= 1) {
        const bool upper = lane & off;
#pragma unroll
        for (int j = 0; j < w / 2; j++) {
            const Sum3 give = upper ? v[j] : v[j + w / 2], keep = upper ? v[j + w / 2] : v[j];
            v[j] = sum_of<THIRD>(keep, shfl_xor_of(give, off));
        }
        if (upper) base += w / 2;
    }
#pragma unroll
    for (int o = off; o > 0; o >>= 1)
        v[0] = o >= 4 ? sum_of<THIRD>(v[0], shfl_xor_of(v[0], o)) : sum_of<true>(v[0], shfl_xor_of(v[0], o));
    if ((lane & (2 * off - 1)) == 0) red[base] = mass_f64(v[0]);
}

// Matrix entries read where they are used: hoisted out of the pass loop, the
// sixteen entries of a dense two-qubit op (96 registers) spill.
template <bool IN_PLACE>
__device__ __forceinline__ void entry(const float4 *w, const float2 *nw, P2 &wr, P2 &wi, P2 &nwi) {
    const uint32_t aw = (uint32_t)__cvta_generic_to_shared(w), an = (uint32_t)__cvta_generic_to_shared(nw);
    if (IN_PLACE) {
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(wr), "=l"(wi) : "r"(aw));
        asm volatile("ld.shared.b64 %0, [%1];" : "=l"(nwi) : "r"(an));
    } else {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(w);
        wr = a.x;
        wi = a.y;
        nwi = *reinterpret_cast<const P2 *>(nw);
    }
}

// Qubits of the op among the lanes of a vector (0, 1) or above.
enum : int { LOW_NONE = 0, LOW_Q0 = 1, LOW_Q1 = 2, LOW_BOTH = 3 };

// A thread's 2^K vectors, two pairs each, as x[j][p]: j the op's qubits, p
// numbering pairs of independent groups. Above the lanes a vector is a
// coordinate and its halves the pairs, as loaded; an op qubit among the lanes
// takes its coordinate from the lane (qubit 1: the vector's halves, qubit 0:
// the lanes of a half), and a vector bit numbers pairs instead.
__device__ __forceinline__ void lanes_2x2(P2 &a, P2 &b) {  // (a0 a1) (b0 b1) -> (a0 b0) (a1 b1)
    const float2 x = pk_float2(a), y = pk_float2(b);
    a = p2_make(x.x, y.x);
    b = p2_make(x.y, y.y);
}
__device__ __forceinline__ void p2_swap(P2 &a, P2 &b) {
    const P2 t = a;
    a = b;
    b = t;
}
template <int K, bool IN>
__device__ __forceinline__ void lanes(P2 (&x)[1 << K][2], int low) {
    constexpr int D = 1 << K;
    if (low == LOW_NONE) return;
    if (K == 2 && low == LOW_BOTH) {  // lane j of vectors 2p, 2p + 1 <-> x[j][p]
#pragma unroll
        for (int i = 0; i < 2; i++)  // order of the two steps is reversed on the way out
            if ((i == 0) == IN) {
#pragma unroll
                for (int p = 0; p < D / 2; p++)
#pragma unroll
                    for (int e = 0; e < 2; e++) lanes_2x2(x[2 * p][e], x[(2 * p + 1) % D][e]);
            } else {
                // (2p + l, e) holds lane 2e + l of pair p: move to (2e + l, p)
                p2_swap(x[0][1], x[2 % D][0]);
                p2_swap(x[1][1], x[3 % D][0]);
            }
        return;
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
        if ((i == 0) == IN) {
            if (low == LOW_Q0) {
#pragma unroll
                for (int v = 0; v < D; v++) lanes_2x2(x[v][0], x[v][1]);
            }
        } else {
            // half e of vector (p, h) <-> x[e | h][p]
#pragma unroll
            for (int h = 0; h < D; h += 2) p2_swap(x[h][1], x[h + 1][0]);
        }
}

// One op's pass for a K-qubit op (K = 1, 2): a thread loads 2^K vectors (four
// groups), scales them by the pending factors, applies the gate and
// accumulates |amplitude|^2 per group coordinate into the warp's table.
// MONO: every matrix row has one entry (CX, SWAP, phases, Pauli strings) and
// no qubit is among the lanes: row r loads its column's vector. The skipped
// terms are exact zeros, so the values are those of the dense sum.
template <int K, bool MONO, int NT, bool SMEM>
__device__ __forceinline__ void traj_pass_body(float *work, uint32_t n, int o, int cur, bool acc) {
    Shared<NT> &s = shared_of<NT>();
    const StateMem<SMEM> sm(work, n);
    constexpr int D = 1 << K;
    const uint32_t q0 = s.op(o).qs[0], q1 = s.op(o).qs[1];
    const int low = MONO || q0 >= 2 ? LOW_NONE : K == 2 && q1 == 1 ? LOW_BOTH : q0 == 0 ? LOW_Q0 : LOW_Q1;
    // the vector bits the thread's vectors span: the op's qubits above the
    // lanes, else the highest free ones (so a warp's loads stay contiguous)
    uint32_t pos[2] = {q0 - 2, q1 - 2};
    if (K == 1) {
        if (low) pos[0] = n - 3;
    } else if (low == LOW_BOTH) {
        pos[0] = n - 4;
        pos[1] = n - 3;
    } else if (low) {  // bit 0 of v numbers groups, bit 1 is qs[1]
        pos[0] = pos[1] == n - 3 ? n - 4 : n - 3;
    }
    const uint32_t plo = K == 1 ? pos[0] : min(pos[0], pos[1]), phi = K == 1 ? 0 : max(pos[0], pos[1]);
    const float4 *W = s.w[cur];
    const float2 *NW = s.nw[cur];
    int col[D];
    if (MONO) {
#pragma unroll
        for (int r = 0; r < D; r++) col[r] = (int)((s.op(o).cols >> (3 * (r ^ s.xm[cur]))) & 7u);
    }
    const int nfv = s.nfv;
    // factor index bits; qubits that are not there read bit 31 of the vector
    // number, which is zero
    const uint32_t fq0 = nfv > 0 ? s.fqv[0] : 31, fq1 = nfv > 1 ? s.fqv[1] : 31, fq2 = nfv > 2 ? s.fqv[2] : 31;
    // Sums per row and lane. With 64 threads the two pairs of groups have one
    // each: as many partial sums, so as small an error, as 256 threads have.
    constexpr int S = NT == 64 ? 2 : 1;
    P2 h[S][D], l[S][D];
#pragma unroll
    for (int i = 0; i < S; i++)
#pragma unroll
        for (int r = 0; r < D; r++) h[i][r] = l[i][r] = 0ull;
    // the thread's vectors: unit u spread around the spanned bits, then those
    auto vector = [&](uint32_t u, int v) {
        uint32_t vb = ((u >> plo) << (plo + 1)) | (u & ((1u << plo) - 1));
        if (K == 2) vb = ((vb >> phi) << (phi + 1)) | (vb & ((1u << phi) - 1));
        uint32_t vi = vb | ((uint32_t)(v & 1) << pos[0]);
        if (K == 2) vi |= (uint32_t)(v >> 1) << pos[1];
        return vi;
    };
    auto source = [&](int v) { return MONO ? col[v] : v; };
    const uint32_t units = 1u << (n - 2 - K);
#pragma unroll 1
    for (uint32_t u = threadIdx.x; u < units; u += NT) {
        P2 xr[D][2], xi[D][2];
#pragma unroll
        for (int v = 0; v < D; v++) {
            const uint32_t vi = vector(u, source(v));
            const ulonglong2 a = *sm.re4(vi), c = *sm.im4(vi);
            xr[v][0] = a.x;
            xr[v][1] = a.y;
            xi[v][0] = c.x;
            xi[v][1] = c.y;
        }
        if (nfv >= 0) {  // factors are real: flips and damping have real operators
#pragma unroll
            for (int v = 0; v < D; v++) {
                const uint32_t vi = vector(u, source(v));
                uint32_t j = ((vi >> fq0) & 1u) | (((vi >> fq1) & 1u) << 1);
                if (nfv > 2) j |= ((vi >> fq2) & 1u) << 2;
                const ulonglong2 f = *reinterpret_cast<const ulonglong2 *>(&s.ft[j]);
                xr[v][0] = p2_mul(f.x, xr[v][0]);
                xr[v][1] = p2_mul(f.y, xr[v][1]);
                xi[v][0] = p2_mul(f.x, xi[v][0]);
                xi[v][1] = p2_mul(f.y, xi[v][1]);
            }
        }
        if (!MONO) {
            lanes<K, true>(xr, low);
            lanes<K, true>(xi, low);
        }
        // one pair of groups at a time, results over the inputs they came from
#pragma unroll
        for (int p = 0; p < 2; p++) {
            P2 br[D], bi[D];
#pragma unroll
            for (int r = 0; r < D; r++) {
                P2 wr, wi, nwi;
                if (MONO) {
                    entry<(K > 1)>(&W[r * D + col[r]], &NW[r * D + col[r]], wr, wi, nwi);
                    br[r] = p2_fma(wr, xr[r][p], p2_mul(nwi, xi[r][p]));
                    bi[r] = p2_fma(wr, xi[r][p], p2_mul(wi, xr[r][p]));
                } else {
#pragma unroll
                    for (int c = 0; c < D; c++) {
                        entry<(K > 1)>(&W[r * D + c], &NW[r * D + c], wr, wi, nwi);
                        const P2 ar = xr[c][p], ai = xi[c][p];
                        br[r] = p2_fma(wr, ar, c ? p2_fma(nwi, ai, br[r]) : p2_mul(nwi, ai));
                        bi[r] = p2_fma(wr, ai, c ? p2_fma(wi, ar, bi[r]) : p2_mul(wi, ar));
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < D; r++) {
                xr[r][p] = br[r];
                xi[r][p] = bi[r];
            }
        }
        if (acc) {  // one branch for all rows: one per row kept their arithmetic apart (126 -> 118 ms)
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int r = 0; r < D; r++)
                    if (NT >= 256) mass_add_pair<MassF2>(xr[r][p], xi[r][p], h[p % S][r], l[p % S][r]);
                    else mass_add2<MassF2>(xr[r][p], xi[r][p], h[p % S][r], l[p % S][r]);
        }
        if (!MONO) {
            lanes<K, false>(xr, low);
            lanes<K, false>(xi, low);
        }
#pragma unroll
        for (int v = 0; v < D; v++) {
            const uint32_t vi = vector(u, v);
            *sm.re4(vi) = make_ulonglong2(xr[v][0], xr[v][1]);
            *sm.im4(vi) = make_ulonglong2(xi[v][0], xi[v][1]);
        }
        if ((u / NT) % (kMassFold / 4) == kMassFold / 4 - 1) {  // four squares per row, lane and unit
#pragma unroll
            for (int i = 0; i < S; i++)
#pragma unroll
                for (int r = 0; r < D; r++) mass_fold<MassF2>(h[i][r], l[i][r]);
        }
    }
    if (!acc) return;
    Sum3 tab[D];
#pragma unroll
    for (int r = 0; r < D; r++) {
        tab[r] = mass_end<(NT < 256)>(h[0][r], l[0][r]);
        if (S == 2) tab[r] = sum_of<true>(tab[r], mass_end<true>(h[S - 1][r], l[S - 1][r]));
    }
    warp_table<D, NT>(tab, s.red[threadIdx.x / 32]);
}

// A dense two-qubit op's pass, out of line: its registers would crowd the
// common passes (one-qubit ops, CX) out of theirs.
template <int NT, bool SMEM>
__device__ __noinline__ void traj_pass_dense2(float *work, uint32_t n, int o, int cur, bool acc) {
    traj_pass_body<2, false, NT, SMEM>(work, n, o, cur, acc);
}

// The general pass, element by element: three-qubit ops and states of fewer
// than five or more than 31 qubits.
template <int NT, bool SMEM>
__device__ __noinline__ void traj_pass_general(float *work, uint32_t n, int o, int cur, bool table) {
    Shared<NT> &s = shared_of<NT>();
    const StateMem<SMEM> sm(work, n);
    const uint64_t len = 1ull << n;
    const uint32_t k = s.op(o).k, dim = 1u << k;
    // Sums per row, for CTAs of up to 128 threads two: a thread's groups in turn.
    constexpr int S = NT <= 128 ? 2 : 1;
    float h[S][8], l[S][8];
#pragma unroll
    for (int i = 0; i < S; i++)
#pragma unroll
        for (int r = 0; r < 8; r++) h[i][r] = l[i][r] = 0.f;
    const uint64_t groups = len >> k;
    auto group = [&](uint64_t g, float (&hs)[8], float (&ls)[8]) {
        const uint64_t base = insert_zeros(g, s.op(o).qs, (int)k);
        float xr[8], xi[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {
            if (j >= dim) break;
            uint64_t idx = base;
            for (uint32_t b = 0; b < k; b++) idx |= (uint64_t)((j >> b) & 1) << s.op(o).qs[b];
            const float f = diag_factor(s, idx);
            xr[j] = f * sm.re(idx);
            xi[j] = f * sm.im(idx);
        }
#pragma unroll
        for (uint32_t r = 0; r < 8; r++) {
            if (r >= dim) break;
            float yr = 0.f, yi = 0.f;
#pragma unroll
            for (uint32_t c = 0; c < 8; c++) {
                if (c >= dim) break;
                const float wr = s.w[cur][r * dim + c].x, wi = s.w[cur][r * dim + c].z;
                yr = fmaf(wr, xr[c], fmaf(-wi, xi[c], yr));
                yi = fmaf(wr, xi[c], fmaf(wi, xr[c], yi));
            }
            uint64_t idx = base;
            for (uint32_t b = 0; b < k; b++) idx |= (uint64_t)((r >> b) & 1) << s.op(o).qs[b];
            sm.re(idx) = yr;
            sm.im(idx) = yi;
            mass_add2<MassF1>(yr, yi, hs[r], ls[r]);
        }
        if ((g / NT) % (kMassFold / 2) >= kMassFold / 2 - S) {
#pragma unroll
            for (int r = 0; r < 8; r++) mass_fold<MassF1>(hs[r], ls[r]);
        }
    };
    for (uint64_t g = threadIdx.x; g < groups; g += S * NT) {
        group(g, h[0], l[0]);
        if (S == 2 && g + NT < groups) group(g + NT, h[S - 1], l[S - 1]);
    }
    if (!table) return;
    Sum3 tab[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < S; i++) {
            mass_fold<MassF1>(h[i][r], l[i][r]);
            const Sum3 x{h[i][r], l[i][r], 0.f};
            tab[r] = i ? sum_of<true>(tab[r], x) : x;
        }
    }
    if (k == 1) warp_table<2, NT>(tab, s.red[threadIdx.x / 32]);
    else if (k == 2) warp_table<4, NT>(tab, s.red[threadIdx.x / 32]);
    else warp_table<8, NT>(tab, s.red[threadIdx.x / 32]);
}

// One warp: the next 32 Philox blocks of trajectory t, one per lane, when
// fewer than 32 are held.
template <int NT>
__device__ __forceinline__ void refill(Shared<NT> &s, uint64_t seed, uint64_t t) {
    __syncwarp();
    if (s.drawn - s.draw < 32) {
        const uint64_t i = s.drawn + threadIdx.x % 32;
        s.us[i % kDraws] = philox_f64(seed, t, i);
        const PhiloxU4 b = philox_block(seed, t, i);
        s.zw[i % kDraws] = ((uint64_t)b.z << 32) | b.w;
        __syncwarp();
        if (threadIdx.x % 32 == 0) s.drawn += 32;
    }
    __syncwarp();
}
template <int NT>
__device__ __forceinline__ double next_f64(Shared<NT> &s) {
    return s.us[s.draw++ % kDraws];
}

// One warp: op `op`'s matrix (gate x the depolarizing string drawn for it,
// draws from stream position `draw` on) into buffer `buf`. Returns the draws
// taken.
template <int NT>
__device__ int prepare_matrix(Shared<NT> &s, const TrajRec &rec, int buf, uint64_t draw, const float *mats,
                              const TrajNoise &nz) {
    const int lane = threadIdx.x % 32;
    const TrajOp &op = rec.op;
    const uint32_t k = op.k, dim = 1u << k;
    uint32_t idx = 0;
    int taken = 0;
    if (op.kind == TOP_GATE && nz.on(k == 1 ? 0 : 1)) {
        taken = 1;
        if (s.us[draw % kDraws] < nz.p[k == 1 ? 0 : 1]) {
            taken = 2;
            idx = 1 + (uint32_t)(((unsigned __int128)s.zw[(draw + 1) % kDraws] * ((1ull << (2 * k)) - 1)) >> 64);
        }
    }
    // P_string . M: the Pauli string is a signed permutation, row r
    // holding its one entry in column r ^ xm (X and Y flip the bit),
    // of value prod_b v_b(r_b) (Y: -i on 0, i on 1; Z: -1 on 1)
    uint32_t xm = 0;
    for (uint32_t b = 0; idx && b < k; b++) {
        const uint32_t code = (idx >> (2 * b)) & 3u;
        if (code == 1 || code == 2) xm |= 1u << b;
    }
    const float *M = k <= 2 ? rec.m : mats + op.mat_off;
    for (uint32_t i = lane; i < dim * dim; i += 32) {
        const uint32_t r = i >> k, c = i & (dim - 1), j = r ^ xm;
        int re_sign = 1, swap = 0;  // phase = re_sign * (swap ? i : 1)
        for (uint32_t b = 0; idx && b < k; b++) {
            const uint32_t code = (idx >> (2 * b)) & 3u, rb = (r >> b) & 1u;
            if (code == 2) {  // multiply by -i (rb = 0) or i (rb = 1)
                if (swap) re_sign = rb ? -re_sign : re_sign;  // i * i = -1, i * -i = 1
                else re_sign = rb ? re_sign : -re_sign;
                swap ^= 1;
            } else if (code == 3 && rb) {
                re_sign = -re_sign;
            }
        }
        const float mr = M[2 * (j * dim + c)], mi = M[2 * (j * dim + c) + 1];
        // (re_sign * (swap ? i : 1)) * (mr + i mi)
        const float wr = swap ? -re_sign * mi : re_sign * mr, wi = swap ? re_sign * mr : re_sign * mi;
        s.w[buf][i] = make_float4(wr, wr, wi, wi);
        s.nw[buf][i] = make_float2(-wi, -wi);
    }
    if (lane == 0) s.xm[buf] = xm;
    return taken;
}

__device__ __forceinline__ bool op_runs(const TrajOp &op, uint64_t cl) {
    if (!op.cond) return true;
    const uint64_t mask = op.cond_len >= 64 ? ~0ull : ((1ull << op.cond_len) - 1);
    return ((cl >> op.cond_off) & mask) == op.cond_value;
}

// Warp 1, during the pass of gate o: copy record o + 2 in, draw ahead, and
// prepare op o + 1, all of which the pass's result has no part in. (What a
// measurement decides, and ops behind one whose condition fails, is left to
// next_op.)
template <int NT>
__device__ __noinline__ void look_ahead(int o, int cur, const TrajRec *recs, int nops, const float *mats,
                                        const TrajNoise &nz, uint64_t seed, uint64_t t) {
    Shared<NT> &s = shared_of<NT>();
    const int lane = threadIdx.x % 32;
    if (o + 2 < nops && lane < (int)(sizeof(TrajRec) / 16))
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(reinterpret_cast<char *>(&s.recs[(o + 2) & 3]) + 16 * lane)),
                     "l"(reinterpret_cast<const char *>(recs + o + 2) + 16 * lane)
                     : "memory");
    refill(s, seed, t);
    const TrajRec &next = s.recs[(o + 1) & 3];
    const bool gate = s.op(o).kind == TOP_GATE;
    int look = LOOK_NO, taken = 0;
    if (gate && o + 1 < nops && op_runs(next.op, s.cl)) {
        // gates take a known number of draws behind their pass
        const int before = s.op(o).k * (nz.on(2) + nz.on(3) + nz.on(4));
        taken = prepare_matrix(s, next, cur ^ 1, s.draw + before, mats, nz);
        look = before ? LOOK_READY : LOOK_GO;
    }
    __syncwarp();
    if (lane == 0) {
        s.look[o & 1] = look;
        s.look_draws = taken;
        if (look == LOOK_GO) s.draw += taken;
    }
}

// Warp 0: the next op that runs, from o on, and its matrix (what look_ahead
// could not do). Records o and o + 1 are held already if `held`.
template <int NT>
__device__ __noinline__ void next_op(int o, int buf, bool held, const TrajRec *recs, int nops, const float *mats,
                                     const TrajNoise &nz) {
    Shared<NT> &s = shared_of<NT>();
    const int lane = threadIdx.x;
    constexpr int kWords = (int)(sizeof(TrajRec) / 4);
    for (;; o++, held = false) {
        __syncwarp();
        for (int r = o; !held && r < o + 2 && r < nops; r++)
            for (int i = lane; i < kWords; i += 32)
                reinterpret_cast<uint32_t *>(&s.recs[r & 3])[i] = reinterpret_cast<const uint32_t *>(recs + r)[i];
        __syncwarp();
        if (o >= nops || op_runs(s.recs[o & 3].op, s.cl)) break;
    }
    int taken = 0;
    if (o < nops) taken = prepare_matrix(s, s.recs[o & 3], buf, s.draw, mats, nz);
    __syncwarp();
    if (lane == 0) {
        s.o = o;
        s.cur = buf;
        s.draw += taken;
    }
    __syncwarp();
}

// Warp 0 after a pass: the flips and damping of a K-qubit gate, resolved on
// the joint table J in the reference's order; the operators are left pending
// (diagonal ones as factors). Every lane computes the same in registers: the
// whole CTA waits for this chain, and a dependent FP64 operation takes 64
// cycles.
template <int K, int NT>
__device__ __forceinline__ void resolve_gate(Shared<NT> &s, int o, const double *Jin, const TrajNoise &nz) {
    constexpr int D = 1 << K;
    double J[D];
#pragma unroll
    for (int j = 0; j < D; j++) J[j] = Jin[j];
    uint64_t draw = s.draw;
    uint32_t q[3] = {0, 0, 0};
    float f0[3] = {1.f, 1.f, 1.f}, f1[3] = {1.f, 1.f, 1.f};
    int nd = 0, np = 0;
    uint32_t qs[K];
#pragma unroll
    for (int b = 0; b < K; b++) qs[b] = s.op(o).qs[b];
#pragma unroll
    for (int b = 0; b < K; b++) {
        float m0 = 1.f, m1 = 0.f, m2 = 0.f, m3 = 1.f;  // row-major, real
        if (nz.on(2) && s.us[draw++ % kDraws] < nz.p[2]) {  // X
            m0 = m3 = 0.f;
            m1 = m2 = 1.f;
#pragma unroll
            for (int j = 0; j < D; j++)
                if (!((j >> b) & 1)) {
                    const double x = J[j];
                    J[j] = J[j | (1 << b)];
                    J[j | (1 << b)] = x;
                }
        }
        if (nz.on(3) && s.us[draw++ % kDraws] < nz.p[3]) {  // Z
            m2 = -m2;
            m3 = -m3;
        }
        if (nz.on(4)) {
            const double u = s.us[draw++ % kDraws];
            // mass0, mass1: of the qubit's two values; P(1) = mass1 / tot
            double mass0 = J[0], mass1 = J[1 << b];
#pragma unroll
            for (int j = 1; j < D; j++)
                if (j != (1 << b)) {
                    if ((j >> b) & 1) mass1 += J[j];
                    else mass0 += J[j];
                }
            const double tot = mass0 + mass1, jump = nz.p[4] * mass1;
            if (u * tot < jump) {
                // jump: collapse to 1 (scale 1/sqrt(P1)) then X
                const float sc = (float)(1.0 / sqrt(mass1 / tot));
                m0 = sc * m2;
                m1 = sc * m3;
                m2 = m3 = 0.f;
#pragma unroll
                for (int j = 0; j < D; j++)
                    if (!((j >> b) & 1)) {
                        J[j] = J[j | (1 << b)] * tot / mass1;
                        J[j | (1 << b)] = 0.0;
                    }
            } else {
                // 1 / sqrt(1 - gamma P(1)) in one rsqrt
                const double sc = tot > 0.0 ? tot * rsqrt((tot - jump) * tot) : 1.0;
                const float k0 = (float)sc, k1 = (float)(sc * s.keep);
                m0 *= k0;
                m1 *= k0;
                m2 *= k1;
                m3 *= k1;
                if (b + 1 < K) {  // the next qubit's masses; the common sc^2 cancels
#pragma unroll
                    for (int j = 0; j < D; j++)
                        if ((j >> b) & 1) J[j] *= s.keep2;
                }
            }
        }
        if (m1 == 0.f && m2 == 0.f) {
            q[nd] = qs[b];
            f0[nd] = m0;
            f1[nd++] = m3;
        } else {
            if (threadIdx.x == 0) s.pend[np] = Pending{qs[b], {{m0, 0}, {m1, 0}, {m2, 0}, {m3, 0}}};
            np++;
        }
    }
    factor_tables(s, nd, q, f0, f1);
    if (threadIdx.x == 0) {
        s.npend = np;
        s.draw = draw;
    }
}

// The same for a three-qubit gate (rare): thread 0, on s.J.
template <int NT>
__device__ __noinline__ void resolve_gate3(int o, const TrajNoise &nz) {
    Shared<NT> &s = shared_of<NT>();
    if (threadIdx.x == 0) {
        const TrajOp &op = s.op(o);
        s.npend = 0;
        for (uint32_t b = 0; b < 3; b++) {
            C2 M[4];
            pauli(0, M);
            if (nz.on(2) && next_f64(s) < nz.p[2]) {
                C2 X[4];
                pauli(1, X);
                mul22(X, M, M);
                for (uint32_t j = 0; j < 8; j++)
                    if (!((j >> b) & 1)) {
                        const double x = s.J[j];
                        s.J[j] = s.J[j | (1u << b)];
                        s.J[j | (1u << b)] = x;
                    }
            }
            if (nz.on(3) && next_f64(s) < nz.p[3]) {
                C2 Z[4];
                pauli(3, Z);
                mul22(Z, M, M);
            }
            if (nz.on(4)) {
                const double u = next_f64(s);
                double mass0 = 0.0, mass1 = 0.0;
                for (uint32_t j = 0; j < 8; j++)
                    if ((j >> b) & 1) mass1 += s.J[j];
                    else mass0 += s.J[j];
                const double tot = mass0 + mass1, jump = nz.p[4] * mass1;
                C2 D[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
                if (u * tot < jump) {
                    D[1] = C2{(float)(1.0 / sqrt(mass1 / tot)), 0};
                    for (uint32_t j = 0; j < 8; j++)
                        if (!((j >> b) & 1)) {
                            s.J[j] = s.J[j | (1u << b)] * tot / mass1;
                            s.J[j | (1u << b)] = 0.0;
                        }
                } else {
                    const double sc = tot > 0.0 ? tot * rsqrt((tot - jump) * tot) : 1.0;
                    D[0] = C2{(float)sc, 0};
                    D[3] = C2{(float)(sc * s.keep), 0};
                    for (uint32_t j = 0; j < 8; j++)
                        if ((j >> b) & 1) s.J[j] *= s.keep2;
                }
                mul22(D, M, M);
            }
            Pending &P = s.pend[s.npend++];
            P.q = op.qs[b];
            for (int i = 0; i < 4; i++) P.m[i] = M[i];
        }
    }
    __syncwarp();
    split_pending(s);
}

// Warp 0 after a measure or reset's pass: the outcome from the table, the
// collapse (and X) left pending.
template <int NT>
__device__ __forceinline__ void resolve_measure(Shared<NT> &s, int o, double J0, double J1, const TrajNoise &nz) {
    const TrajOp &op = s.op(o);
    uint64_t draw = s.draw;
    const double tot = J0 + J1;
    const bool one = s.us[draw++ % kDraws] * tot < J1;  // u < P(1), src/exec.rs:201-207
    const float sc = (float)(tot * rsqrt((one ? J1 : J0) * tot));  // 1 / sqrt(P(outcome))
    const uint32_t q[3] = {op.qs[0], 0, 0};
    const bool flip = one && op.kind == TOP_RESET;  // X . diag(0, sc)
    const float f0[3] = {one ? 0.f : sc, 1.f, 1.f}, f1[3] = {one ? sc : 0.f, 1.f, 1.f};
    factor_tables(s, flip ? 0 : 1, q, f0, f1);
    uint64_t cl = s.cl;
    if (op.kind == TOP_MEASURE) {
        bool bit = one;
        const double pr = bit ? nz.p[6] : nz.p[5];  // readout_flip (src/noise.rs:181-192)
        if (nz.on(bit ? 6 : 5) && s.us[draw++ % kDraws] < pr) bit = !bit;
        cl = (cl & ~(1ull << op.clbit)) | ((uint64_t)bit << op.clbit);
    }
    __syncwarp();
    if (threadIdx.x == 0) {
        if (flip) s.pend[0] = Pending{op.qs[0], {{0, 0}, {sc, 0}, {0, 0}, {0, 0}}};
        s.npend = flip;
        s.cl = cl;
        s.draw = draw;
    }
}

// Warp 0 behind a pass of a K-qubit op: the CTA's table from the warps'
// (lanes in groups of NW, each summing one entry or every 32 / NW-th), the
// op's noise or outcome, and the step to the next op.
template <int K, int NT>
__device__ __noinline__ void finish_op(int o, int cur, bool acc, const TrajRec *recs, int nops, const float *mats,
                                       const TrajNoise &nz) {
    constexpr int NW = NT / 32, G = 32 / NW, D = 1 << K;
    Shared<NT> &s = shared_of<NT>();
    const int lane = threadIdx.x;
    double J[D];
#pragma unroll
    for (int j = 0; j < D; j++) J[j] = 0.0;
    if (acc) {
        double v[D];
#pragma unroll
        for (int j = 0; j < D; j += G) v[j] = s.red[lane % NW][(j + lane / NW) & (D - 1)];
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < D; j += G) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
#pragma unroll
        for (int j = 0; j < D; j++) J[j] = __shfl_sync(0xffffffffu, v[j - j % G], (j % G) * NW);
    }
    const bool gate = s.op(o).kind == TOP_GATE;
    if constexpr (K == 3) {
#pragma unroll
        for (int j = 0; j < D; j++) s.J[j] = J[j];  // every lane the same
        __syncwarp();
        resolve_gate3<NT>(o, nz);
    } else {
        if (gate) resolve_gate<K>(s, o, J, nz);
        else resolve_measure(s, o, J[0], J[1], nz);
    }
    __syncwarp();
    const int look = s.look[o & 1];
    if (look != LOOK_NO) {
        if (lane == 0) {
            if (look == LOOK_READY) s.draw += s.look_draws;
            s.o = o + 1;
            s.cur = cur ^ 1;
        }
    } else {
        next_op<NT>(o + 1, cur ^ 1, true, recs, nops, mats, nz);
    }
}

// |a|^2 of element i with the pending factors, as f64.
template <int NT, bool SMEM>
__device__ __forceinline__ double mass_at(const StateMem<SMEM> &sm, const Shared<NT> &s, uint64_t i) {
    const float f = diag_factor(s, i), xr = f * sm.re(i), xi = f * sm.im(i);
    return (double)xr * xr + (double)xi * xi;
}

// Warp: the mass of elements [i0, i1).
template <int NT, bool SMEM>
__device__ double range_mass(const StateMem<SMEM> &sm, const Shared<NT> &s, uint64_t i0, uint64_t i1) {
    P2 h[2] = {0, 0}, l[2] = {0, 0};  // a lane's elements in turn
    const uint64_t first = i0 + threadIdx.x % 32;
    auto value = [&](uint64_t i) {
        if (i >= i1) return MassF2::zero();
        const float f = diag_factor(s, i);
        return p2_make(f * sm.re(i), f * sm.im(i));
    };
    uint32_t folded = 0;
    for (uint64_t i = first; i < i1; i += 128) {
        mass_add2<MassF2>(value(i), value(i + 64), h[0], l[0]);
        mass_add2<MassF2>(value(i + 32), value(i + 96), h[1], l[1]);
        if (++folded == kMassFold / 2) {
            folded = 0;
#pragma unroll
            for (int j = 0; j < 2; j++) mass_fold<MassF2>(h[j], l[j]);
        }
    }
    Sum3 v = sum_of<true>(mass_end<true>(h[0], l[0]), mass_end<true>(h[1], l[1]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = sum_of<true>(v, shfl_xor_of(v, o));
    return mass_f64(v);
}

// One basis index from |psi|^2 by the draw u in [0, 1): region (one per
// warp), block (32 per region) and element whose cumulative mass first
// exceeds it. Left in s.u's stead as an index in every thread.
template <int NT, bool SMEM>
__device__ __noinline__ uint64_t sample_index(float *work, uint32_t n) {
    Shared<NT> &s = shared_of<NT>();
    const StateMem<SMEM> sm(work, n);
    const uint64_t len = 1ull << n;
    constexpr int NW = NT / 32;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint64_t W = (len + NW - 1) / NW, B = (W + 31) / 32;  // elements per region, per block
    const uint64_t w0 = min(len, warp * W), w1 = min(len, w0 + W);
    const double seg = range_mass(sm, s, w0, w1);
    if (lane == 0) s.seg[warp] = seg;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int i = 0; i < NW; i++) tot += s.seg[i];
        double u = next_f64(s) * tot;
        int r = 0;
        while (r < NW && !(u < s.seg[r])) u -= s.seg[r++];
        s.region = r;
        s.u = u;
    }
    __syncthreads();
    const int region = s.region;
    uint64_t pick = len;
    if (region < NW) {
        const uint64_t r0 = min(len, region * W), r1 = min(len, r0 + W);
        for (int b = warp; b < 32; b += NW) {
            const uint64_t b0 = min(r1, r0 + b * B), b1 = min(r1, b0 + B);
            const double m = range_mass(sm, s, b0, b1);
            if (lane == 0) s.blk[b] = m;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double u = s.u;
            int b = 0, last = 0;
            for (; b < 32 && !(u < s.blk[b]); b++) {
                if (s.blk[b] > 0.0) last = b;
                u -= s.blk[b];
            }
            s.block = b < 32 ? b : last;  // rounding past the region's end: its last block with mass
            s.u = b < 32 ? u : __longlong_as_double(0x7ff0000000000000ll);
        }
        __syncthreads();
        // the block's elements, in order, 1024 at a time
        const uint64_t b0 = min(r1, r0 + s.block * B), b1 = min(r1, b0 + B);
        double u = s.u;
        bool found = false;
        for (uint64_t c0 = b0; c0 < b1 && !found; c0 += 1024) {
            const uint64_t c1 = min(b1, c0 + 1024);
            __syncthreads();
            for (uint64_t i = c0 + threadIdx.x; i < c1; i += NT) s.el[i - c0] = mass_at(sm, s, i);
            __syncthreads();
            if (threadIdx.x == 0) {
                for (uint64_t i = c0; i < c1; i++) {
                    const double p = s.el[i - c0];
                    if (p > 0.0) pick = i;  // last nonzero so far
                    if (u < p) {
                        found = true;
                        break;
                    }
                    u -= p;
                }
            }
            found = __syncthreads_or(found);
        }
    }
    if (threadIdx.x == 0 && pick == len) {
        // rounding left the draw past the last region: last index with nonzero probability
        pick = 0;
        for (uint64_t i = len; i-- > 0;)
            if (mass_at(sm, s, i) > 0.0) {
                pick = i;
                break;
            }
    }
    return pick;  // thread 0's counts
}

// NT threads per CTA. SMEM: the whole state in shared memory (ns unused).
template <int NT, int CTAS, bool SMEM>
__global__ void __launch_bounds__(NT, CTAS)
    k_trajectories(float *__restrict__ work, uint32_t n, const TrajRec *__restrict__ recs, int nops,
                   const float *__restrict__ mats, const uint32_t *__restrict__ fq, const uint32_t *__restrict__ fc,
                   int nfinal, TrajNoise nz, uint64_t ntraj, uint64_t seed, uint64_t *__restrict__ out) {
    Shared<NT> &s = shared_of<NT>();
    const uint64_t len = 1ull << n;
    if (!SMEM) work += (size_t)blockIdx.x * 2 * len;
    const StateMem<SMEM> sm(work, n);
    const int tid = threadIdx.x, warp = tid / 32;
    const bool vec = n >= 5 && n <= 31;
    if (tid == 0) {
        s.keep = sqrt(1.0 - nz.p[4]);
        s.keep2 = s.keep * s.keep;
    }
    for (uint64_t t = blockIdx.x; t < ntraj; t += gridDim.x) {
        for (uint64_t i = tid; i < len; i += NT) {
            sm.re(i) = i == 0 ? 1.f : 0.f;
            sm.im(i) = 0.f;
        }
        if (warp == 0) {
            const uint32_t q[3] = {0, 0, 0};
            const float f[3] = {1.f, 1.f, 1.f};
            factor_tables(s, 0, q, f, f);
            if (tid == 0) {
                s.npend = 0;
                s.draw = s.drawn = 0;
                s.cl = 0;
            }
            refill(s, seed, t);
            next_op<NT>(0, 0, false, recs, nops, mats, nz);
        }
        __syncthreads();
        int o = s.o, cur = s.cur;
        while (o < nops) {
            const bool factors = s.npend || s.nfv >= 0;
            if (s.npend) apply_nondiag_pending<NT, SMEM>(work, n);
            const uint32_t k = s.op(o).k;
            const bool acc = wants_table(s.op(o), nz);
            if (warp == 1) look_ahead<NT>(o, cur, recs, nops, mats, nz, seed, t);
            const bool mono = s.op(o).mono && s.op(o).qs[0] >= 2;
            if (!vec || k > 2) traj_pass_general<NT, SMEM>(work, n, o, cur, acc);
            else if (k == 1 && !mono) traj_pass_body<1, false, NT, SMEM>(work, n, o, cur, acc);
            else if (k == 1) traj_pass_body<1, true, NT, SMEM>(work, n, o, cur, acc);
            else if (mono) traj_pass_body<2, true, NT, SMEM>(work, n, o, cur, acc);
            else traj_pass_dense2<NT, SMEM>(work, n, o, cur, acc);
            if (warp == 1) asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // nothing to decide and nothing pending before or after: on to the
            // next pass with this one barrier
            if (s.look[o & 1] == LOOK_GO && !factors) {
                o++;
                cur ^= 1;
                continue;
            }
            if (warp == 0) {
                if (k == 1) finish_op<1, NT>(o, cur, acc, recs, nops, mats, nz);
                else if (k == 2) finish_op<2, NT>(o, cur, acc, recs, nops, mats, nz);
                else finish_op<3, NT>(o, cur, acc, recs, nops, mats, nz);
            }
            __syncthreads();
            o = s.o;
            cur = s.cur;
        }
        // ---- final: pending operators, then one basis index from |psi|^2
        if (s.npend) apply_nondiag_pending<NT, SMEM>(work, n);
        if (warp == 0) refill(s, seed, t);
        const uint64_t pick = sample_index<NT, SMEM>(work, n);
        if (warp == 0) {
            uint64_t cl = s.cl;
            for (int f = 0; f < nfinal; f++) {
                refill(s, seed, t);
                if (tid == 0) {
                    bool bit = (pick >> fq[f]) & 1;
                    const double pr = bit ? nz.p[6] : nz.p[5];
                    if (nz.on(bit ? 6 : 5) && next_f64(s) < pr) bit = !bit;
                    cl = (cl & ~(1ull << fc[f])) | ((uint64_t)bit << fc[f]);
                }
            }
            if (tid == 0) out[t] = cl;
        }
        __syncthreads();
    }
}

template <int NT, int CTAS, bool SMEM>
int run_trajectories(zc_state *st, const TrajPlan &plan, uint32_t n, const TrajRec *d_recs, int nops,
                     const float *d_mats, const uint32_t *d_fq, const uint32_t *d_fc, int nfinal, const TrajNoise &nz,
                     uint64_t ntraj, uint64_t seed, uint64_t *d_out, float *d_work) {
    ZC_CUDA(cudaFuncSetAttribute(k_trajectories<NT, CTAS, SMEM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kTrajSmemMax));
    k_trajectories<NT, CTAS, SMEM><<<plan.ctas, NT, plan.smem, st->stream>>>(
        d_work, n, d_recs, nops, d_mats, d_fq, d_fc, nfinal, nz, ntraj, seed, d_out);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

}  // namespace

// CTA size and placement by state size (f32, 8 bytes per amplitude), 128
// registers per thread everywhere:
//   <= 10 qubits (8 KiB)    64 threads, eight per SM: a pass is a few vectors
//                           per thread, latency is hidden across trajectories
//   <= 12 qubits (32 KiB)   128 threads, four per SM
//   13 qubits (64 KiB)      256 threads, two per SM; all these in shared memory
//   14 qubits (128 KiB)     512 threads, one per SM, all in shared memory
//   above                   512 threads, one per SM, the first 24576
//                           amplitudes in shared memory, the rest in global
TrajPlan plan_trajectories(uint32_t n, uint64_t ntraj, int num_sms) {
    TrajPlan p{};
    const uint64_t len = 1ull << n;
    p.threads = n <= 10 ? 64 : n <= 12 ? 128 : n == 13 ? 256 : 512;
    p.smem = std::min<uint64_t>(len, kTrajSplitElems) * 8;
    p.global_bytes = n <= 14 ? 0 : len * 8;
    p.ctas = (int)std::min<uint64_t>(ntraj, (uint64_t)num_sms * (512 / p.threads));
    return p;
}

int launch_trajectories(zc_state *st, const TrajPlan &plan, uint32_t n, const TrajRec *d_recs, int nops,
                        const float *d_mats, const uint32_t *d_fq, const uint32_t *d_fc, int nfinal,
                        const TrajNoise &nz, uint64_t ntraj, uint64_t seed, uint64_t *d_out, void *d_work) {
    ProfScope ps(st, K_TRAJ, 0.0);
    st->ctr.launches++;
    if (st->prec != 32) return fail(ZC_ERR_UNSUPPORTED, "the batched trajectory engine runs f32 states");
    auto run = plan.threads == 64    ? run_trajectories<64, 8, true>
               : plan.threads == 128 ? run_trajectories<128, 4, true>
               : plan.threads == 256 ? run_trajectories<256, 2, true>
                                     : run_trajectories<512, 1, false>;
    return run(st, plan, n, d_recs, nops, d_mats, d_fq, d_fc, nfinal, nz, ntraj, seed, d_out, (float *)d_work);
}

}  // namespace zc
