// Multi-op sweep kernel: one pass over HBM applies a whole run of ops.
//
// The state is cut into tiles of 2^T amplitudes: the L lowest qubits (a
// contiguous row of 2^L elements, 256 bytes) plus H chosen higher qubits
// ("local" qubits); the other n - T qubits pick the tile. A persistent CTA
// streams tiles through one shared-memory buffer: a tile is fetched with
// asynchronous 16-byte copies, the sweep's micro-ops are applied in shared
// memory, and it goes back with 16-byte stores; three CTAs per SM overlap one
// tile's copies with the others' arithmetic. In exact mode every micro-op uses the
// same arithmetic as the per-op kernels, so a sweep is bit-identical to
// launching its ops one by one; fast f64 sweeps run the lowered ops
// (zc_lower.cpp) in register passes of packed double-float arithmetic.
//
// Which ops fit a sweep: unitaries whose qubits are all local; diagonals
// on any qubits (bits of non-local qubits are constant per tile); CX with a
// local target and any control; SWAP of two local qubits.
#include <string.h>

#include <algorithm>
#include <atomic>

#include "zc_arith.cuh"
#include "zc_async.cuh"
#include "zc_internal.h"
#include "zc_passes.h"
#include "zc_sweep.h"

namespace zc {
namespace {

constexpr int kSweepThreads = 256;  // table diagonals split an index at its eighth bit
constexpr int kSweepCtasPerSm = 3;
// The tile's re array, then, this far behind it whatever the tile's size, im.
constexpr uint32_t kTileArrayBytes = (uint32_t)(kSweepSmemBytes / 2);

// Where element v of a tile array of ES-byte elements sits: 16-byte vectors
// stay whole and in their 128-byte row, and the vector's place in the row is
// XORed with higher index bits. A pass that pairs low index bits otherwise
// reads with power-of-two strides and hits the same banks: conflicts were
// 30-45% of the shared-memory wavefronts of a sweep, and those wavefronts are
// what bounds it (65-84% of peak). The map is linear over XOR and its own
// inverse: swz(a ^ b) = swz(a) ^ swz(b), swz(swz(v)) = v.
template <int ES>
__host__ __device__ __forceinline__ uint32_t swz(uint32_t v) {
    constexpr uint32_t VB = ES == 4 ? 2 : ES == 8 ? 1 : 0;  // elements per vector, log2 (16: vectors themselves)
    return v ^ ((((v >> (VB + 3)) ^ (v >> (VB + 6))) & 7u) << VB);
}

// Global index of the first element of tile t: the tile number fills the
// non-local positions above the L low bits.
__device__ __forceinline__ uint64_t tile_base(uint64_t t, uint32_t L, const uint32_t *hpos, uint32_t H) {
    return insert_zeros(t << L, hpos, (int)H);
}

// Swap the slots v0 <-> v1 of both arrays (values of any representation).
template <typename T>
__device__ __forceinline__ void swap_slots(T *sr, T *si, uint32_t v0, uint32_t v1) {
    T x = sr[v0];
    sr[v0] = sr[v1];
    sr[v1] = x;
    x = si[v0];
    si[v0] = si[v1];
    si[v1] = x;
}

// Swap 16-byte vectors of slots (VW consecutive elements) at v0 <-> v1.
__device__ __forceinline__ void swap_vec(void *sr, void *si, uint32_t v0, uint32_t v1) {
    uint4 *r = reinterpret_cast<uint4 *>(sr), *i = reinterpret_cast<uint4 *>(si);
    const uint4 a = r[v0], b = r[v1], c = i[v0], d = i[v1];
    r[v0] = b;
    r[v1] = a;
    i[v0] = d;
    i[v1] = c;
}

__host__ __device__ __forceinline__ uint32_t insert_zero32(uint32_t v, uint32_t b) {
    return ((v >> b) << (b + 1)) | (v & ((1u << b) - 1));
}

// Permutation micro-ops (CX, SWAP) move raw slots, so they serve every
// arithmetic policy and representation. When none of the op's bits is among
// the lowest log2(VW), the VW consecutive slots of a 16-byte vector move
// together: one vector load and store per VW elements.
template <typename T>
__device__ void apply_perm(T *sr, T *si, const OpHead &op, uint64_t base, uint32_t size) {
    const int tid = threadIdx.x, nt = blockDim.x;
    constexpr uint32_t VW = 16 / sizeof(T), VB = VW == 4 ? 2 : 1;  // elements per vector, log2
    const uint32_t nv = size / VW;                                   // vectors in the tile
    constexpr int ES = (int)sizeof(T);
    if (op.kind == MOP_CX && !(op.a & kOuterFlag) && min(op.a, op.b) >= VB) {
        const uint32_t c = op.a - VB, t = op.b - VB, lo = min(c, t), hi = max(c, t);
        const uint32_t ct = swz<16>(1u << c), tt = swz<16>(1u << t);
        for (uint32_t p = tid; p < nv / 4; p += nt) {
            const uint32_t v0 = swz<16>(insert_zero32(insert_zero32(p, lo), hi)) ^ ct;
            swap_vec(sr, si, v0, v0 ^ tt);
        }
        return;
    }
    if (op.kind == MOP_CX && (op.a & kOuterFlag) && op.b >= VB) {
        if (!((base >> (op.a & ~kOuterFlag)) & 1)) return;
        const uint32_t t = op.b - VB, tt = swz<16>(1u << t);
        for (uint32_t p = tid; p < nv / 2; p += nt) {
            const uint32_t v0 = swz<16>(insert_zero32(p, t));
            swap_vec(sr, si, v0, v0 ^ tt);
        }
        return;
    }
    if (op.kind == MOP_SWAP && min(op.a, op.b) >= VB) {
        const uint32_t lo = min(op.a, op.b) - VB, hi = max(op.a, op.b) - VB;
        const uint32_t tl = swz<16>(1u << lo), th = swz<16>(1u << hi);
        for (uint32_t p = tid; p < nv / 4; p += nt) {
            const uint32_t v = swz<16>(insert_zero32(insert_zero32(p, lo), hi));
            swap_vec(sr, si, v ^ tl, v ^ th);
        }
        return;
    }
    if (op.kind == MOP_CX) {
        const uint32_t t = op.b, tt = swz<ES>(1u << t);
        if (op.a & kOuterFlag) {
            if (!((base >> (op.a & ~kOuterFlag)) & 1)) return;
            for (uint32_t p = tid; p < size / 2; p += nt) {
                const uint32_t v0 = swz<ES>(insert_zero32(p, t));
                swap_slots(sr, si, v0, v0 ^ tt);
            }
        } else {
            const uint32_t c = op.a, lo = min(c, t), hi = max(c, t), ct = swz<ES>(1u << c);
            for (uint32_t p = tid; p < size / 4; p += nt) {
                const uint32_t v0 = swz<ES>(insert_zero32(insert_zero32(p, lo), hi)) ^ ct;
                swap_slots(sr, si, v0, v0 ^ tt);
            }
        }
    } else {
        const uint32_t lo = min(op.a, op.b), hi = max(op.a, op.b);
        const uint32_t tl = swz<ES>(1u << lo), th = swz<ES>(1u << hi);
        for (uint32_t p = tid; p < size / 4; p += nt) {
            const uint32_t v = swz<ES>(insert_zero32(insert_zero32(p, lo), hi));
            swap_slots(sr, si, v ^ tl, v ^ th);
        }
    }
}

// Per-op coefficients in the compute representation, as encode_job leaves them.
// U1: the 2x2 matrix; D1: entries 0..3 = d0r d0i d1r d1i. Double-float
// pairs for A == AR_DF, else values of T. Double-float RT: v[0] = t, and
// v[2..6) its packed pairs (PkReal: t hi, t lo, -t hi, -t lo, each twice).
template <typename T, int A>
struct alignas(16) OpCoef {
    typename std::conditional<A == AR_DF, float2, T>::type v[8];
};

// The packed pairs of a double-float rotation's t, read where the rotation
// runs: hoisted above a group's amplitude loads, the pairs of three
// rotations (24 registers) spill at the 80-register cap.
template <typename T, int A>
__device__ __forceinline__ PkReal rot_pairs(const OpCoef<T, A> &c) {
    float4 a, b;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
                 : "r"(smem_addr(&c.v[2])));
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "r"(smem_addr(&c.v[4])));
    return PkReal{make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
}

// Double-float sweeps hold each amplitude as packed pairs: slot v of the
// re array H = (re hi, im hi), of the im array L = (re lo, im lo). General
// gates use the scalar routines on split pairs.
__device__ __forceinline__ void hl_rdf(const float2 *r, float2 &Ha, float2 &La, float2 &Hb, float2 &Lb) {
    float2 ar, ai, br, bi;
    pk_split(Ha, La, ar, ai);
    pk_split(Hb, Lb, br, bi);
    pair_update_rdf(r, ar, ai, br, bi);
    pk_join(ar, ai, Ha, La);
    pk_join(br, bi, Hb, Lb);
}
__device__ __forceinline__ void hl_udf(const MatDF &m, float2 &Ha, float2 &La, float2 &Hb, float2 &Lb) {
    float2 ar, ai, br, bi;
    pk_split(Ha, La, ar, ai);
    pk_split(Hb, Lb, br, bi);
    pair_update_df(m, ar, ai, br, bi);
    pk_join(ar, ai, Ha, La);
    pk_join(br, bi, Hb, Lb);
}
// Diagonals outside register passes take normalised pairs (the product drops lo x
// lo, which after a chain of unnormalised rotations is no longer below the last
// bit: 20-qubit QFT off by 8.4e-15 so, 1.1e-14 without, in the same time) and
// leave them unnormalised, as register passes do: the ops after them accept
// that, and the sweep's exit renormalises.
__device__ __forceinline__ void hl_cscale_df(float2 wr, float2 wi, float2 &H, float2 &L) {
    float2 ar, ai;
    pk_renorm(H, L);
    pk_split(H, L, ar, ai);
    cscale_df_u(wr, wi, ar, ai);
    pk_join(ar, ai, H, L);
}

// The register group size of double-float sweeps: they spill at the
// 80-register cap with more than two general ops (rotations: three).
constexpr int kDfGroup = 2;
// The pass descriptors of a job, one slot per op (exact f64 sweeps have none).
template <typename T, int A>
struct PassOf {
    using type = typename std::conditional<A == AR_DF, GroupInfo, RegOp>::type;
    static constexpr bool any = A == AR_DF || sizeof(T) == 4;
};

__device__ __forceinline__ uint32_t jouter(const OpHead &op, uint64_t base) {
    uint32_t jo = 0;
    for (uint32_t b = 0; b < op.k; b++)
        if (op.loc[b] & kOuterFlag) jo |= (uint32_t)((base >> (op.loc[b] & ~kOuterFlag)) & 1) << b;
    return jo;
}

// One pass (see GroupInfo) of a double-float sweep. xr / xi hold the packed
// pairs H / L; the rotations run as f32x2 arithmetic.
// Every index a thread needs (its slot, its load slot under the folded CX
// block, its table entry) is linear over XOR in the group number p, so it is
// worked out once per pass, as byte offsets, and a group of three bits (two
// groups per thread) steps to its second group by XORing the descriptor's
// step patterns; the im array sits a fixed distance behind re. Index work was
// half of a pass's instructions when it was redone per group and element.
// in_f64 / out_f64: the slots hold f64 on entry / must hold f64 on exit (the
// sweep's first / last pass does the tile's conversion in registers).
template <typename T, int A, int G, bool ROT_ONLY, bool HAS_DK, bool HAS_CX>
__device__ void run_pass(const GroupInfo &gi, char *tile, const OpHead *ops, const OpCoef<T, A> *coef, uint32_t size,
                         const char *tables, uint64_t base, bool in_f64, bool out_f64) {
    constexpr int E = 1 << G;
    const int o = gi.first;
    uint32_t jo = 0, u0 = 0;
    if constexpr (HAS_DK) {
        for (int i = 0; i < gi.nout; i++) jo |= (uint32_t)((base >> gi.outq[i]) & 1u) << (gi.outb[i] + 4);
    }
    if constexpr (HAS_CX) {
        for (int t = 0; t < gi.ntr; t++)
            if ((gi.trc[t] & 0x80u) && ((base >> (gi.trc[t] & 0x7fu)) & 1u)) u0 ^= gi.trw[t];
    }
    uint32_t so = 0, lo = 0, jb = 0;  // slot, load slot, table entry of element 0, in bytes
    for (uint32_t p = threadIdx.x; p < size / E; p += kSweepThreads) {
        if (G == 3 && p >= kSweepThreads) {  // at most one step: tiles have 2^12 elements
            so ^= gi.so_step;
            lo ^= gi.lo_step;
            jb ^= gi.jb_step;
        } else {
            uint32_t v = p;
#pragma unroll
            for (int g = 0; g < G; g++) v = insert_zero32(v, gi.sorted[g]);
            so = lo = swz<8>(v) << 3;
            if constexpr (HAS_CX) {  // the descriptor's slot patterns are byte offsets of swizzled slots
                lo ^= u0;
                for (int t = 0; t < gi.ntr; t++)
                    if (!(gi.trc[t] & 0x80u) && ((v >> gi.trc[t]) & 1u)) lo ^= gi.trw[t];
            }
            if constexpr (HAS_DK) {
                jb = jo;
                for (int i = 0; i < gi.nloc; i++) jb |= ((v >> gi.loc[i]) & 1u) << (gi.locb[i] + 4);
            }
        }
        float2 xr[E], xi[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            uint32_t w = lo;
#pragma unroll
            for (int g = 0; g < G; g++)
                if ((e >> g) & 1) w ^= HAS_CX ? gi.pm[g] : gi.gm[g];
            if (in_f64) {
                pk_from_f64(*reinterpret_cast<const double *>(tile + w),
                            *reinterpret_cast<const double *>(tile + kTileArrayBytes + w), xr[e], xi[e]);
            } else {
                xr[e] = *reinterpret_cast<const float2 *>(tile + w);
                xi[e] = *reinterpret_cast<const float2 *>(tile + kTileArrayBytes + w);
            }
        }
        if constexpr (HAS_DK) {
            const char *dtab = tables + gi.tab_off;
            uint32_t tm[G];
#pragma unroll
            for (int g = 0; g < G; g++) tm[g] = gi.tb[g] != 0xff ? 16u << gi.tb[g] : 0u;
#pragma unroll
            for (int e = 0; e < E; e++) {
                uint32_t j = jb;
#pragma unroll
                for (int g = 0; g < G; g++)
                    if ((e >> g) & 1) j ^= tm[g];
                const float4 w = __ldg(reinterpret_cast<const float4 *>(dtab + j));
                float2 ar, ai;  // scalar: the packed form needs eight registers per entry
                pk_split(xr[e], xi[e], ar, ai);
                cscale_df_u(make_float2(w.x, w.y), make_float2(w.z, w.w), ar, ai);
                pk_join(ar, ai, xr[e], xi[e]);
            }
        }
        // the diagonal and the rotations chain unnormalised pairs (every
        // double-float op accepts them; |lo| grows by about an ulp of hi per
        // op, so the absolute error stays at the double-float bound);
        // renormalised only where the tile goes back to f64
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (ROT_ONLY || ops[o + g].kind == MOP_RT) {
                const PkReal t = rot_pairs(coef[o + g]);
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (!((e >> g) & 1)) pk_rot_u(t, xr[e], xi[e], xr[e | (1 << g)], xi[e | (1 << g)]);
            } else if (ops[o + g].kind == MOP_R1) {
                float2 r[4];
#pragma unroll
                for (int i = 0; i < 4; i++) r[i] = coef[o + g].v[i];
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (!((e >> g) & 1)) hl_rdf(r, xr[e], xi[e], xr[e | (1 << g)], xi[e | (1 << g)]);
            } else {
                MatDF m;
#pragma unroll
                for (int i = 0; i < 8; i++) m.v[i] = coef[o + g].v[i];
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (!((e >> g) & 1)) hl_udf(m, xr[e], xi[e], xr[e | (1 << g)], xi[e | (1 << g)]);
            }
        }
        const uint32_t fo = so ^ gi.fmask;
#pragma unroll
        for (int e = 0; e < E; e++) {
            uint32_t w = fo;
#pragma unroll
            for (int g = 0; g < G; g++)
                if ((e >> g) & 1) w ^= gi.gm[g];
            if (out_f64) {
                pk_to_f64(xr[e], xi[e], *reinterpret_cast<double *>(tile + w),
                          *reinterpret_cast<double *>(tile + kTileArrayBytes + w));
            } else {  // the next pass accepts unnormalised pairs
                *reinterpret_cast<float2 *>(tile + w) = xr[e];
                *reinterpret_cast<float2 *>(tile + kTileArrayBytes + w) = xi[e];
            }
        }
    }
}

// One gate of an f32 pass on the group coordinate G.
template <int G, bool EXACT>
__device__ __forceinline__ void reg_gate(const Mat2<float> &m, float *xr, float *xi) {
#pragma unroll
    for (int e = 0; e < 1 << kRegBits; e++)
        if (!((e >> G) & 1)) pair_update<float, EXACT>(m, xr[e], xi[e], xr[e | (1 << G)], xi[e | (1 << G)]);
}

// The CX with target coordinate G: pairs whose bit of `on` is set change places.
template <int G>
__device__ __forceinline__ void reg_cx(uint32_t on, float *xr, float *xi) {
#pragma unroll
    for (int e = 0; e < 1 << kRegBits; e++) {
        constexpr int F = 1 << G;
        if ((e >> G) & 1) continue;
        const bool sw = (on >> e) & 1u;
        const float ar = xr[e], ai = xi[e], br = xr[e | F], bi = xi[e | F];
        xr[e] = sw ? br : ar;
        xi[e] = sw ? bi : ai;
        xr[e | F] = sw ? ar : br;
        xi[e | F] = sw ? ai : bi;
    }
}

// A pass of an f32 sweep (RegOp): its ops in order on sixteen elements in
// registers, one round trip through shared memory for all of them. The
// wavefronts of a trip per op (per pair of gates) bound f32 sweeps; four bits
// take four to five ops of a random circuit. Out of line: inlined into the tile
// loop it spilled at the 80-register cap. Bound by instruction issue now (69%
// of the slots at three CTAs per SM; f32x2 gates took 18% of the instructions
// away and no time). 26 qubits, random gates: 17.2 -> 16.0 ms, 24 packed states
// of 8 to 22 qubits 7.8 -> 7.4 (10.9 with a trip per pair of gates).
template <typename T, int A>
__device__ __noinline__ void run_pass_f32(const RegOp *pass, const OpHead *ops, const OpCoef<T, A> *coef, char *tile,
                                          uint32_t size, const char *tables, uint64_t base) {
    constexpr int E = 1 << kRegBits;
    constexpr bool EX = A == AR_EXACT;
    const int n = pass[0].n;
    for (uint32_t p = threadIdx.x; p < size / E; p += kSweepThreads) {
        uint32_t v = p, gm[kRegBits];
#pragma unroll
        for (int g = 0; g < kRegBits; g++) {
            v = insert_zero32(v, pass[0].sorted[g]);
            gm[g] = swz<4>(1u << pass[0].sorted[g]) << 2;
        }
        const uint32_t so = swz<4>(v) << 2;
        auto slot = [&](int e) {
            uint32_t w = so;
#pragma unroll
            for (int g = 0; g < kRegBits; g++)
                if ((e >> g) & 1) w ^= gm[g];
            return w;
        };
        float xr[E], xi[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const uint32_t w = slot(e);
            xr[e] = *reinterpret_cast<const float *>(tile + w);
            xi[e] = *reinterpret_cast<const float *>(tile + kTileArrayBytes + w);
        }
        // bit of location l (a tile bit outside the group, or an outer qubit)
        auto bit_of = [&](uint32_t l) {
            return (l & kOuterFlag) ? (uint32_t)(base >> (l & ~kOuterFlag)) & 1u : (v >> l) & 1u;
        };
        // elements whose selecting bit is set
        auto chosen = [&](uint32_t c, uint32_t l) {
            return c != 0xffu ? (uint32_t)(0xff00f0f0ccccaaaaull >> (16 * c)) & 0xffffu : 0u - bit_of(l);
        };
#pragma unroll 1
        for (int k = 0; k < n; k++) {
            const RegOp &r = pass[k];
            const OpHead &op = ops[k];
            if (op.kind == MOP_U1) {
                Mat2<float> m;
#pragma unroll
                for (int i = 0; i < 8; i++) m.v[i] = coef[k].v[i];
                if (r.g == 0) reg_gate<0, EX>(m, xr, xi);
                else if (r.g == 1) reg_gate<1, EX>(m, xr, xi);
                else if (r.g == 2) reg_gate<2, EX>(m, xr, xi);
                else reg_gate<3, EX>(m, xr, xi);
            } else if (op.kind == MOP_CX) {
                const uint32_t on = chosen(r.c, op.a);
                if (r.g == 0) reg_cx<0>(on, xr, xi);
                else if (r.g == 1) reg_cx<1>(on, xr, xi);
                else if (r.g == 2) reg_cx<2>(on, xr, xi);
                else reg_cx<3>(on, xr, xi);
            } else if (op.kind == MOP_D1) {
                const uint32_t on = chosen(r.c, op.a);
                const float d0r = coef[k].v[0], d0i = coef[k].v[1], d1r = coef[k].v[2], d1i = coef[k].v[3];
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const bool one = (on >> e) & 1u;
                    cscale<float, EX>(one ? d1r : d0r, one ? d1i : d0i, xr[e], xi[e]);
                }
            } else {
                uint32_t j = 0;
                for (uint32_t b = 0; b < op.k; b++)
                    if (!((r.tm[0] | r.tm[1] | r.tm[2] | r.tm[3]) >> b & 1u)) j |= bit_of(op.loc[b]) << b;
                const float2 *tab = reinterpret_cast<const float2 *>(tables + op.table);
#pragma unroll
                for (int e = 0; e < E; e++) {
                    uint32_t i = j;
#pragma unroll
                    for (int g = 0; g < kRegBits; g++)
                        if ((e >> g) & 1) i |= r.tm[g];
                    const float2 w = __ldg(tab + i);
                    cscale<float, EX>(w.x, w.y, xr[e], xi[e]);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
            const uint32_t w = slot(e);
            *reinterpret_cast<float *>(tile + w) = xr[e];
            *reinterpret_cast<float *>(tile + kTileArrayBytes + w) = xi[e];
        }
    }
}

template <typename T, int A, int G, bool ROT_ONLY>
__device__ void run_pass_any(const GroupInfo &gi, char *tile, const OpHead *ops,
                             const OpCoef<T, A> *coef, uint32_t size, const char *tables, uint64_t base, bool in_f64,
                             bool out_f64) {
    const bool cx = gi.ntr || gi.pm[0] != gi.gm[0] || (G > 1 && gi.pm[G - 1] != gi.gm[G - 1]) ||
                    (G > 2 && gi.pm[1] != gi.gm[1]);
    if (gi.has_dk) {
        if (cx) run_pass<T, A, G, ROT_ONLY, true, true>(gi, tile, ops, coef, size, tables, base, in_f64, out_f64);
        else run_pass<T, A, G, ROT_ONLY, true, false>(gi, tile, ops, coef, size, tables, base, in_f64, out_f64);
    } else {
        if (cx) run_pass<T, A, G, ROT_ONLY, false, true>(gi, tile, ops, coef, size, tables, base, in_f64, out_f64);
        else run_pass<T, A, G, ROT_ONLY, false, false>(gi, tile, ops, coef, size, tables, base, in_f64, out_f64);
    }
}

// gis: the job's register passes (double-float and f32 sweeps);
// fuse_in / fuse_out: its first / last pass converts the tile.
template <typename T, int A, typename R>
__device__ void apply_ops(R *sr, R *si, const OpHead *ops, const OpCoef<T, A> *coef, int nops, uint64_t base,
                          uint32_t size, const char *tables,
                          const typename PassOf<T, A>::type *gis,
                          int fuse_in = 0, int fuse_out = 0) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int o = 0; o < nops; o++) {
        const OpHead &op = ops[o];
        if constexpr (A == AR_DF) {
            const GroupInfo &gi = gis[o];
            if (gi.G) {
                const bool in_f64 = o == 0 && fuse_in, out_f64 = o + gi.skip == nops && fuse_out;
                if (gi.rot3)
                    run_pass_any<T, A, 3, true>(gi, reinterpret_cast<char *>(sr), ops, coef, size, tables, base, in_f64, out_f64);
                else if (gi.G == 2)
                    run_pass_any<T, A, 2, false>(gi, reinterpret_cast<char *>(sr), ops, coef, size, tables, base, in_f64, out_f64);
                else
                    run_pass_any<T, A, 1, false>(gi, reinterpret_cast<char *>(sr), ops, coef, size, tables, base, in_f64, out_f64);
                o += gi.skip - 1;
                __syncthreads();
                continue;
            }
        }
        if constexpr (sizeof(T) == 4) {
            const int n = gis[o].n;
            if (n) {
                run_pass_f32<T, A>(gis + o, ops + o, coef + o, reinterpret_cast<char *>(sr), size, tables, base);
                o += n - 1;
                __syncthreads();
                continue;
            }
        }
        // one gate: exact f64 (~400 integer instructions per pair hide the
        // trip), and f32 states smaller than a pass's bits
        if constexpr (A != AR_DF) {
            if (op.kind == MOP_U1) {
                const uint32_t b = op.a, bs = swz<(int)sizeof(R)>(1u << b);
                if constexpr (A == AR_EXACT && sizeof(T) == 8) {
                    const double *m = coef[o].v;
                    const ExactMask mask = exact_mask(m);
#pragma unroll 1
                    for (uint32_t p = tid; p < size / 2; p += nt) {
                        const uint32_t v0 = swz<(int)sizeof(R)>(insert_zero32(p, b)), v1 = v0 ^ bs;
                        double ar = sr[v0], ai = si[v0], br = sr[v1], bi = si[v1];
                        pair_update_f64(m, mask, ar, ai, br, bi);
                        sr[v0] = ar;
                        si[v0] = ai;
                        sr[v1] = br;
                        si[v1] = bi;
                    }
                    __syncthreads();
                    continue;
                }
                Mat2<T> m;
#pragma unroll
                for (int i = 0; i < 8; i++) m.v[i] = coef[o].v[i];
                for (uint32_t p = tid; p < size / 2; p += nt) {
                    const uint32_t v0 = swz<(int)sizeof(R)>(insert_zero32(p, b)), v1 = v0 ^ bs;
                    pair_update<T, A == AR_EXACT>(m, sr[v0], si[v0], sr[v1], si[v1]);
                }
                __syncthreads();
                continue;
            }
        }
        if (op.kind == MOP_D1) {
            const bool outer = op.a & kOuterFlag;
            const bool tile_one = outer && ((base >> (op.a & ~kOuterFlag)) & 1);
            auto scl = [&](uint32_t v, R &xr, R &xi) {
                const bool one = outer ? tile_one : ((v >> op.a) & 1);
                if constexpr (A == AR_DF) hl_cscale_df(coef[o].v[one ? 2 : 0], coef[o].v[one ? 3 : 1], xr, xi);
                else cscale<T, A == AR_EXACT>(coef[o].v[one ? 2 : 0], coef[o].v[one ? 3 : 1], xr, xi);
            };
            uint32_t v = tid;
            for (; v + 3u * nt < size; v += 4u * nt) {
                R xr[4], xi[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    xr[k] = sr[v + k * nt];
                    xi[k] = si[v + k * nt];
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    scl(swz<(int)sizeof(R)>(v + k * nt), xr[k], xi[k]);
                    sr[v + k * nt] = xr[k];
                    si[v + k * nt] = xi[k];
                }
            }
            for (; v < size; v += nt) scl(swz<(int)sizeof(R)>(v), sr[v], si[v]);
        } else if (op.kind == MOP_DK) {
            // The table index of the element in slot v is linear over XOR: the
            // bits of v select masks that the job brings along (in the op's
            // coefficients). Gathering the op's bits through a lookup table
            // built per tile cost the 25-qubit QFT a tenth (10.5 -> 9.5 ms).
            const uint16_t *mask = reinterpret_cast<const uint16_t *>(&coef[o]);
            uint32_t j0 = jouter(op, base);
#pragma unroll
            for (int b = 0; b < 8; b++) j0 ^= (tid >> b) & 1 ? mask[b] : 0u;
            auto index_of = [&](uint32_t v) {
                uint32_t j = j0;
#pragma unroll
                for (int b = 8; b < 13; b++) j ^= (v >> b) & 1u ? mask[b] : 0u;
                return j;
            };
            // (re, im) pairs of T, or double-float (re hi, re lo, im hi, im lo)
            using P2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
            const P2 *ptab = reinterpret_cast<const P2 *>(tables + op.table);
            const float4 *dtab = reinterpret_cast<const float4 *>(tables + op.table);
            // W: the table entry (T re, T im; or one float4 of double-float pairs)
            using W = typename std::conditional<A == AR_DF, float4, T>::type;
            auto load_w = [&](uint32_t j, W &wr, W &wi) {
                if constexpr (A == AR_DF) {
                    wr = __ldg(dtab + j);
                } else {
                    const P2 w = __ldg(ptab + j);
                    wr = w.x;
                    wi = w.y;
                }
            };
            auto scl = [&](const W &wr, const W &wi, R &xr, R &xi) {
                if constexpr (A == AR_DF) hl_cscale_df(make_float2(wr.x, wr.y), make_float2(wr.z, wr.w), xr, xi);
                else cscale<T, A == AR_EXACT>(wr, wi, xr, xi);
            };
            uint32_t v = tid;
            for (; v + 3u * nt < size; v += 4u * nt) {
                R xr[4], xi[4];
                W wr[4], wi[4];
                const uint32_t j = index_of(v);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    load_w(j ^ (k & 1 ? mask[8] : 0u) ^ (k & 2 ? mask[9] : 0u), wr[k], wi[k]);
                    xr[k] = sr[v + k * nt];
                    xi[k] = si[v + k * nt];
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    scl(wr[k], wi[k], xr[k], xi[k]);
                    sr[v + k * nt] = xr[k];
                    si[v + k * nt] = xi[k];
                }
            }
            for (; v < size; v += nt) {
                W wr, wi;
                load_w(index_of(v), wr, wi);
                scl(wr, wi, sr[v], si[v]);
            }
        } else {
            apply_perm(sr, si, op, base, size);
        }
        __syncthreads();
    }
}

// Per-CTA state of a sweep: the current job's micro-ops, coefficients and
// row offsets.
template <typename T, int A>
struct SweepSmem {
    OpHead ops[kMaxMicroOps];
    OpCoef<T, A> coef[kMaxMicroOps];
    uint32_t rows[1u << kMaxSweepHigh];  // row r of a tile starts at element rows[r] << L of it
    JobHead job;
    alignas(16) typename PassOf<T, A>::type gi[PassOf<T, A>::any ? kMaxMicroOps : 1];  // register passes
};
static_assert(sizeof(OpHead[kMaxMicroOps]) % 16 == 0 && sizeof(GroupInfo[kMaxMicroOps]) % 16 == 0,
              "job sections are copied in 16-byte pieces");

// A job's block for the kernel (see JobHead). Everything that depends on the
// job alone is worked out here, once: a CTA of a small or mid-size state has
// one tile, and the passes resolved there by one thread took longer than the
// tile (a 4-qubit double-float sweep: 95 us; a 19-qubit one 52 us).
template <typename T, int A>
int encode_job_as(const SweepPlan &plan, std::vector<char> *out) {
    const int nops = (int)plan.mops.size();
    if (((size_t)2 << (plan.g.L + plan.g.H)) * sizeof(T) > kSweepSmemBytes)
        return fail(ZC_ERR_INVALID, "sweep shape exceeds the kernel's limits");
    JobHead h{};
    h.nops = (uint32_t)nops;
    h.L = plan.g.L;
    h.H = plan.g.H;
    for (uint32_t j = 0; j < h.H && j < 8; j++) h.hpos[j] = plan.g.hpos[j];
    std::vector<OpHead> ops((size_t)nops);
    std::vector<OpCoef<T, A>> coef((size_t)nops);
    for (int o = 0; o < nops; o++) {
        const MicroOp &m = plan.mops[(size_t)o];
        memcpy(&ops[(size_t)o], &m, sizeof(OpHead));
        h.has_arith |= m.kind != MOP_CX && m.kind != MOP_SWAP;
        const int cnt = m.kind == MOP_U1 ? 8 : m.kind == MOP_RT ? 1 : m.kind == MOP_D1 || m.kind == MOP_R1 ? 4 : 0;
        if (!operands_ok(ops[(size_t)o], h.L + h.H, plan.g.n))
            return fail(ZC_ERR_INVALID, "sweep plan: an operand lies outside the tile and the state");
        constexpr size_t entry = A == AR_DF ? 16 : 2 * sizeof(T);
        if (m.kind == MOP_DK && (m.table % 16 || m.table + (entry << m.k) > plan.tables.size()))
            return fail(ZC_ERR_INVALID, "sweep plan: a diagonal lies outside the tables");
        OpCoef<T, A> &c = coef[(size_t)o];
        for (int i = 0; i < cnt; i++) {
            if constexpr (A == AR_DF) {
                const float hi = (float)m.m[i];
                c.v[i] = make_float2(hi, (float)(m.m[i] - (double)hi));
            } else {
                c.v[i] = (T)m.m[i];
            }
        }
        if (m.kind == MOP_DK) {  // table index masks of the slot bits (see apply_ops)
            uint16_t mask[13] = {};
            static_assert(sizeof mask <= sizeof c, "index masks fit the op's coefficients");
            for (uint32_t b = 0; b < h.L + h.H; b++)
                for (uint32_t i = 0; i < m.k; i++)
                    if (!(m.loc[i] & kOuterFlag)) mask[b] |= (uint16_t)(((swz<(int)sizeof(T)>(1u << b) >> m.loc[i]) & 1u) << i);
            memcpy((void *)&c, mask, sizeof mask);
        }
        if constexpr (A == AR_DF) {
            if (m.kind == MOP_RT) {  // the rotation's packed pairs
                const float2 t = c.v[0];
                c.v[2] = make_float2(t.x, t.x);
                c.v[3] = make_float2(t.y, t.y);
                c.v[4] = make_float2(-t.x, -t.x);
                c.v[5] = make_float2(-t.y, -t.y);
            }
        }
    }
    std::vector<typename PassOf<T, A>::type> gi;
    if constexpr (sizeof(T) == 4) {
        gi.resize((size_t)nops);
        plan_reg_passes(ops.data(), nops, h.L + h.H, gi.data());
    }
    if constexpr (A == AR_DF) {
        gi.resize((size_t)nops);
        uint32_t bad = 0;
        int fuse_in = 0, fuse_out = 0;
        plan_passes(ops.data(), nops, h.L + h.H, true, kDfGroup, gi.data(), &bad, &fuse_in, &fuse_out);
        if (bad) return fail(ZC_ERR_INVALID, "sweep plan: a group bit lies outside the tile");
        h.fuse_in = (uint32_t)fuse_in;
        h.fuse_out = (uint32_t)fuse_out;
        for (GroupInfo &q : gi) {  // slot patterns as byte offsets into the swizzled tile, step patterns
            if (!q.G) continue;
            for (int g = 0; g < q.G; g++) {
                q.gm[g] = (uint16_t)(swz<8>(q.gm[g]) << 3);
                q.pm[g] = (uint16_t)(swz<8>(q.pm[g]) << 3);
            }
            for (int i = 0; i < q.ntr; i++) q.trw[i] = (uint16_t)(swz<8>(q.trw[i]) << 3);
            q.fmask = (uint16_t)(swz<8>(q.fmask) << 3);
            uint32_t v = kSweepThreads, lo = 0, jb = 0;  // group number p + kSweepThreads against p
            for (int g = 0; g < q.G; g++) v = insert_zero32(v, q.sorted[g]);
            for (int i = 0; i < q.ntr; i++)
                if (!(q.trc[i] & 0x80u) && ((v >> q.trc[i]) & 1u)) lo ^= q.trw[i];
            for (int i = 0; i < q.nloc; i++) jb |= ((v >> q.loc[i]) & 1u) << (q.locb[i] + 4);
            q.so_step = (uint16_t)(swz<8>(v) << 3);
            q.lo_step = (uint16_t)(q.so_step ^ lo);
            q.jb_step = (uint16_t)jb;
        }
    }
    auto up16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
    const size_t ops_b = up16(ops.size() * sizeof(OpHead)), coef_b = up16(coef.size() * sizeof(OpCoef<T, A>));
    h.coef_off = (uint32_t)(sizeof(JobHead) + ops_b);
    h.gi_off = (uint32_t)(h.coef_off + coef_b);
    out->assign(h.gi_off + up16(gi.size() * sizeof(gi[0])), 0);
    memcpy(out->data(), &h, sizeof h);
    memcpy(out->data() + sizeof(JobHead), ops.data(), ops.size() * sizeof(OpHead));
    memcpy(out->data() + h.coef_off, (const void *)coef.data(), coef.size() * sizeof(OpCoef<T, A>));
    if (!gi.empty()) memcpy(out->data() + h.gi_off, gi.data(), gi.size() * sizeof(gi[0]));
    return ZC_OK;
}

__device__ __forceinline__ void copy16(void *dst, const char *src, uint32_t bytes) {
    for (uint32_t i = threadIdx.x; i < (bytes + 15) / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(dst)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
}

// All threads: make the job block at `blk` the CTA's current job.
template <typename T, int A>
__device__ void load_job(SweepSmem<T, A> &c, const char *blk) {
    const int tid = threadIdx.x;
    const JobHead *h = reinterpret_cast<const JobHead *>(blk);
    const uint32_t nops = h->nops, L = h->L, H = h->H;
    __syncthreads();  // the previous job's tiles are done with the tables
    copy16(&c.job, blk, sizeof(JobHead));
    copy16(c.ops, blk + sizeof(JobHead), nops * (uint32_t)sizeof(OpHead));
    copy16(c.coef, blk + h->coef_off, nops * (uint32_t)sizeof(OpCoef<T, A>));
    if constexpr (PassOf<T, A>::any) copy16(c.gi, blk + h->gi_off, nops * (uint32_t)sizeof(c.gi[0]));
    for (uint32_t r = tid; r < (1u << H); r += blockDim.x) {  // tile bit L + j holds qubit hpos[j]
        uint32_t o = 0;
        for (uint32_t j = 0; j < H; j++) o |= ((r >> j) & 1u) << (h->hpos[j] - L);
        c.rows[r] = o;
    }
    __syncthreads();
}

// All threads: one array of a tile between global and shared memory, 16
// bytes per access (a row is 256 bytes, or less for states under 2^L).
// Loads are asynchronous copies (wait_all, then a barrier); stores go
// through registers, four in flight.
template <typename T, int A>
__device__ __forceinline__ void tile_load(const SweepSmem<T, A> &c, T *dst, const T *src, uint32_t vecs) {
    constexpr uint32_t VW = 16 / sizeof(T), VB = VW == 4 ? 2 : 1;
    const uint32_t lv = c.job.L - VB, cm = (1u << lv) - 1;  // vectors per row (log2), column mask
    const uint32_t d = smem_addr(dst);
    if (c.job.L < VB) {  // a state shorter than one vector
        if (threadIdx.x < (1u << c.job.L)) dst[threadIdx.x] = src[threadIdx.x];
        return;
    }
    for (uint32_t i = threadIdx.x; i < vecs; i += kSweepThreads) {
        const T *g = src + ((size_t)c.rows[i >> lv] << c.job.L) + (size_t)(i & cm) * VW;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * swz<16>(i)), "l"(g) : "memory");
    }
}
template <typename T, int A>
__device__ __forceinline__ void tile_store(const SweepSmem<T, A> &c, T *dst, const T *src, uint32_t vecs) {
    constexpr uint32_t VW = 16 / sizeof(T), VB = VW == 4 ? 2 : 1;
    const uint32_t lv = c.job.L - VB, cm = (1u << lv) - 1;
    if (c.job.L < VB) {
        if (threadIdx.x < (1u << c.job.L)) dst[threadIdx.x] = src[threadIdx.x];
        return;
    }
    const uint4 *sv = reinterpret_cast<const uint4 *>(src);
    auto at = [&](uint32_t i) {
        return reinterpret_cast<uint4 *>(dst + ((size_t)c.rows[i >> lv] << c.job.L) + (size_t)(i & cm) * VW);
    };
    uint32_t i = threadIdx.x;
    for (; i + 3 * kSweepThreads < vecs; i += 4 * kSweepThreads) {
        uint4 x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = sv[swz<16>(i + k * kSweepThreads)];
#pragma unroll
        for (int k = 0; k < 4; k++) *at(i + k * kSweepThreads) = x[k];
    }
    for (; i < vecs; i += kSweepThreads) *at(i) = sv[swz<16>(i)];
}

// All threads: one tile of the current job — load, micro-ops in shared
// memory, store.
// The tile moves by plain 16-byte accesses of all threads (32 per thread and
// tile). One TMA bulk copy per 256-byte row, issued by one warp, kept the
// copy unit busy ~75 cycles per row: 20k cycles for a tile's loads and 22k
// for its stores beside 38k of arithmetic, at three CTAs per SM
// (clock64 at 26 qubits). The same circuits with
// this: 27q depth-10 fast f64 84.3 -> 72.3 ms, 26q f32 gate mix 22.3 -> 18.8.
template <typename T, int A>
__device__ void process_tile(SweepSmem<T, A> &c, T *re, T *im, uint64_t t, const char *tables, T *sre, T *sim,
                             uint32_t form) {
    const uint32_t size = 1u << (c.job.L + c.job.H), vecs = size / (16 / (uint32_t)sizeof(T));
    const int tid = threadIdx.x;
    const uint64_t base = tile_base(t, c.job.L, c.job.hpos, c.job.H);
    tile_load(c, sre, re + base, vecs);
    tile_load(c, sim, im + base, vecs);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if constexpr (A == AR_DF) {
        // The slots hold f64, or (form & kFormInDf) the normalised packed
        // pairs the previous sweep left (re slot H, im slot L); on exit f64,
        // or (form & kFormOutDf) normalised packed pairs. CX / SWAP move slots
        // whatever they hold. Each conversion reads both slots of an element
        // before it writes either.
        double *dr = reinterpret_cast<double *>(sre), *di = reinterpret_cast<double *>(sim);
        float2 *fr = reinterpret_cast<float2 *>(sre), *fi = reinterpret_cast<float2 *>(sim);
        const bool in_df = form & kFormInDf, out_df = form & kFormOutDf;
        const bool fuse_in = c.job.fuse_in && !in_df, fuse_out = c.job.fuse_out && !out_df;
        auto to_pairs = [&](uint32_t v) {
            float2 H, L;
            pk_from_f64(dr[v], di[v], H, L);
            fr[v] = H;
            fi[v] = L;
        };
        auto to_f64 = [&](uint32_t v) {
            double a, b;
            pk_to_f64(fr[v], fi[v], a, b);
            dr[v] = a;
            di[v] = b;
        };
        if (c.job.has_arith && !in_df && !c.job.fuse_in) {
            for (uint32_t v = tid; v < size; v += blockDim.x) to_pairs(v);
            __syncthreads();
        }
        apply_ops<T, A, float2>(fr, fi, c.ops, c.coef, (int)c.job.nops, base, size, tables, c.gi,
                                fuse_in,
                                fuse_out);
        if (c.job.has_arith && !fuse_out) {  // register passes leave pairs unnormalised
            for (uint32_t v = tid; v < size; v += blockDim.x) {
                if (out_df) {
                    float2 H = fr[v], L = fi[v];
                    pk_renorm(H, L);
                    fr[v] = H;
                    fi[v] = L;
                } else {
                    to_f64(v);
                }
            }
        } else if (!c.job.has_arith && in_df != out_df) {  // permutations only: change the form alone
            for (uint32_t v = tid; v < size; v += blockDim.x) {
                if (in_df) to_f64(v);
                else to_pairs(v);
            }
        }
    } else {
        apply_ops<T, A, T>(sre, sim, c.ops, c.coef, (int)c.job.nops, base, size, tables, c.gi);
    }
    __syncthreads();
    tile_store(c, re + base, sre, vecs);
    tile_store(c, im + base, sim, vecs);
    __syncthreads();  // the buffer is free
}

// One state. One CTA streams tiles through a single shared-memory buffer;
// three CTAs per SM overlap one tile's traffic with the others' arithmetic.
// FORM (g.form as a compile-time constant): each hand-over of double-float
// pairs between sweeps is its own instantiation, so the tile loop carries no
// run-time branches for it (they cost registers at the 80-register cap).
template <typename T, int A, uint32_t FORM>
__global__ void __launch_bounds__(kSweepThreads, kSweepCtasPerSm)
    k_sweep(T *__restrict__ re, T *__restrict__ im, uint64_t ntiles, const char *__restrict__ job,
            const char *__restrict__ tables) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ SweepSmem<T, A> c;
    T *sre = reinterpret_cast<T *>(smem);
    T *sim = sre + kTileArrayBytes / sizeof(T);
    load_job(c, job);
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) process_tile(c, re, im, t, tables, sre, sim, FORM);
}

// Many states in one launch (the serving engine's packed step): the tiles
// of all jobs form one index space; a CTA switches job when its next tile
// belongs to another state.
template <typename T, int A>
__global__ void __launch_bounds__(kSweepThreads, kSweepCtasPerSm)
    k_sweep_multi(const char *__restrict__ blob) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ SweepSmem<T, A> c;
    const SweepBatch *hdr = reinterpret_cast<const SweepBatch *>(blob);
    const SweepJob *jobs = reinterpret_cast<const SweepJob *>(blob + sizeof(SweepBatch));
    const uint32_t njobs = hdr->njobs;
    const uint64_t total = hdr->total_tiles;
    int cur = -1;
    // Tiles go to CTAs round-robin (concurrent tiles stay adjacent in memory
    // and big and small jobs mix evenly); the job is looked up only when a
    // tile falls outside the current one.
    uint64_t job_lo = 1, job_hi = 0;
    for (uint64_t t = blockIdx.x; t < total; t += gridDim.x) {
        if (t < job_lo || t >= job_hi) {
            uint32_t lo = 0, hi = njobs;  // last job with tile_start <= t
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (jobs[mid].tile_start <= t) lo = mid;
                else hi = mid;
            }
            const SweepJob &Jn = jobs[lo];
            load_job(c, blob + Jn.job_off);
            cur = (int)lo;
            job_lo = Jn.tile_start;
            job_hi = Jn.tile_start + Jn.ntiles;
        }
        const SweepJob &J = jobs[cur];
        T *sre = reinterpret_cast<T *>(smem);
        T *sim = sre + kTileArrayBytes / sizeof(T);
        process_tile(c, reinterpret_cast<T *>(J.re), reinterpret_cast<T *>(J.im), t - J.tile_start,
                     blob + J.tables_off, sre, sim, 0u);
    }
}

template <typename T, int A, uint32_t FORM>
int run_sweep_form(zc_state *st, const SweepGeom &g, const char *dev_job, const char *dev_tables) {
    static std::atomic<bool> attr{false};  // set once per process; racing first calls repeat it
    if (!attr) {
        ZC_CUDA(cudaFuncSetAttribute(k_sweep<T, A, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSweepSmemBytes));
        attr = true;
    }
    const uint64_t blocks = std::min<uint64_t>(g.ntiles, (uint64_t)st->num_sms * kSweepCtasPerSm);
    k_sweep<T, A, FORM><<<(int)blocks, kSweepThreads, kSweepSmemBytes, st->stream>>>(
        (T *)st->re, (T *)st->im, g.ntiles, dev_job, dev_tables);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

template <typename T, int A>
int run_sweep(zc_state *st, const SweepGeom &g, const char *dev_job, const char *dev_tables) {
    if constexpr (A == AR_DF) {
        switch (g.form) {
            case 0: return run_sweep_form<T, A, 0>(st, g, dev_job, dev_tables);
            case kFormInDf: return run_sweep_form<T, A, kFormInDf>(st, g, dev_job, dev_tables);
            case kFormOutDf: return run_sweep_form<T, A, kFormOutDf>(st, g, dev_job, dev_tables);
            default: return run_sweep_form<T, A, kFormInDf | kFormOutDf>(st, g, dev_job, dev_tables);
        }
    }
    if (g.form) return fail(ZC_ERR_INVALID, "double-float hand-over requested outside a double-float sweep");
    return run_sweep_form<T, A, 0>(st, g, dev_job, dev_tables);
}

template <typename T, int A>
int run_sweep_multi(cudaStream_t stream, int num_sms, const char *dev_blob) {
    static std::atomic<bool> attr{false};  // set once per process; racing first calls repeat it
    if (!attr) {
        ZC_CUDA(cudaFuncSetAttribute(k_sweep_multi<T, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSweepSmemBytes));
        attr = true;
    }
    k_sweep_multi<T, A><<<num_sms * kSweepCtasPerSm, kSweepThreads, kSweepSmemBytes, stream>>>(dev_blob);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

// Round a state that double-float sweeps left as packed pairs (re slot
// H = (re hi, im hi), im slot L = (re lo, im lo)) back to f64 (the last sweep
// of a flush normally does this itself; this pass serves a flush whose
// double-float sweeps are followed by another kernel).
__global__ void __launch_bounds__(256) k_df_to_f64(double *__restrict__ re, double *__restrict__ im, uint64_t len) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = reinterpret_cast<const double2 *>(re)[i];
        const double2 b = reinterpret_cast<const double2 *>(im)[i];
        const float4 fa = *reinterpret_cast<const float4 *>(&a), fb = *reinterpret_cast<const float4 *>(&b);
        double r0, i0, r1, i1;
        pk_to_f64(make_float2(fa.x, fa.y), make_float2(fb.x, fb.y), r0, i0);
        pk_to_f64(make_float2(fa.z, fa.w), make_float2(fb.z, fb.w), r1, i1);
        reinterpret_cast<double2 *>(re)[i] = make_double2(r0, r1);
        reinterpret_cast<double2 *>(im)[i] = make_double2(i0, i1);
    }
}

}  // namespace

int load_sweep_kernels(int prec, bool exact) {
    if (prec == 32) {
        if (exact) ZC_LOAD(k_sweep<float, AR_EXACT, 0>);
        else ZC_LOAD(k_sweep<float, AR_FMA, 0>);
    } else if (exact) {
        ZC_LOAD(k_sweep<double, AR_EXACT, 0>);
    } else {
        ZC_LOAD(k_sweep<double, AR_DF, 0>);
        ZC_LOAD(k_sweep<double, AR_DF, kFormInDf>);
        ZC_LOAD(k_sweep<double, AR_DF, kFormOutDf>);
        ZC_LOAD(k_sweep<double, AR_DF, kFormInDf | kFormOutDf>);
        ZC_LOAD(k_df_to_f64);
    }
    return ZC_OK;
}

int launch_df_to_f64(zc_state *st) {
    ProfScope ps(st, K_SWEEP, 2.0 * st->len * 8 * 2);
    st->ctr.launches++;
    st->ctr.sweeps++;
    st->ctr.bytes_moved += 2 * st->len * 8 * 2;
    const uint64_t n2 = st->len / 2;  // two elements per thread step (sweeps have at least 2^3)
    const uint64_t blocks = std::min<uint64_t>((n2 + 255) / 256, (uint64_t)st->num_sms * 8);
    k_df_to_f64<<<(int)blocks, 256, 0, st->stream>>>((double *)st->re, (double *)st->im, n2);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

int launch_sweep_multi(cudaStream_t stream, int num_sms, int prec, bool exact, const char *dev_blob) {
    if (prec == 64)
        return exact ? run_sweep_multi<double, AR_EXACT>(stream, num_sms, dev_blob)
                     : run_sweep_multi<double, AR_DF>(stream, num_sms, dev_blob);
    return exact ? run_sweep_multi<float, AR_EXACT>(stream, num_sms, dev_blob)
                 : run_sweep_multi<float, AR_FMA>(stream, num_sms, dev_blob);
}

int encode_job(int prec, bool exact, const SweepPlan &plan, std::vector<char> *out) {
    if (plan.mops.size() > (size_t)kMaxMicroOps || plan.g.H > kMaxSweepHigh)
        return fail(ZC_ERR_INVALID, "sweep shape exceeds the kernel's limits");
    if (prec == 64) return exact ? encode_job_as<double, AR_EXACT>(plan, out) : encode_job_as<double, AR_DF>(plan, out);
    return exact ? encode_job_as<float, AR_EXACT>(plan, out) : encode_job_as<float, AR_FMA>(plan, out);
}

int launch_sweep(zc_state *st, const SweepGeom &g, const char *dev_job, const char *dev_tables, bool exact) {
    ProfScope ps(st, K_SWEEP, 2.0 * st->len * (st->prec / 8) * 2);
    st->ctr.launches++;
    st->ctr.sweeps++;
    st->ctr.bytes_moved += 2 * st->len * (st->prec / 8) * 2;
    if (st->prec == 64)
        return exact ? run_sweep<double, AR_EXACT>(st, g, dev_job, dev_tables)
                     : run_sweep<double, AR_DF>(st, g, dev_job, dev_tables);
    return exact ? run_sweep<float, AR_EXACT>(st, g, dev_job, dev_tables)
                 : run_sweep<float, AR_FMA>(st, g, dev_job, dev_tables);
}

}  // namespace zc
