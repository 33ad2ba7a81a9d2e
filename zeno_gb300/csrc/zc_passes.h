// Register passes of double-float and f32 sweeps: the micro-op head the tile loop
// reads, the pass descriptor and the planning of the passes of a job. Shared
// by the sweep kernel (zc_sweep.cu) and the host check of the pass logic
// (tests/passes_harness.cpp).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "zc_sweep.h"

#ifdef __CUDACC__
#define ZC_HD __host__ __device__ __forceinline__
#else
#define ZC_HD inline
#endif

namespace zc {

constexpr int kMaxFoldCx = 4;  // CX ops one register group takes into its loads

// The part of a MicroOp the tile loop reads (its first 72 bytes); the matrix
// entries go into the job's coefficients.
struct OpHead {
    uint32_t kind, a, b, k;
    uint32_t loc[12];
    uint64_t table;
};
static_assert(sizeof(OpHead) == 72 && offsetof(MicroOp, table) == offsetof(OpHead, table) &&
                  offsetof(MicroOp, m) == sizeof(OpHead),
              "OpHead is the head of MicroOp");

// Whether the kernel can run an op on a tile of 2^tile_log2 slots of an n-qubit
// state: every operand a tile bit or, where that is allowed, an outer qubit.
// The kernel indexes shared memory with them unchecked.
inline bool operands_ok(const OpHead &op, uint32_t tile_log2, uint32_t n) {
    auto local = [&](uint32_t x) { return x < tile_log2; };
    auto any = [&](uint32_t x) { return (x & kOuterFlag) ? (x & ~kOuterFlag) < n : local(x); };
    switch (op.kind) {
        case MOP_U1:
        case MOP_R1:
        case MOP_RT: return local(op.a);
        case MOP_D1: return any(op.a);
        case MOP_DK:
            if (op.k < 1 || op.k > 12) return false;
            for (uint32_t b = 0; b < op.k; b++)
                if (!any(op.loc[b])) return false;
            return true;
        case MOP_CX: return any(op.a) && local(op.b) && op.a != op.b;
        case MOP_SWAP: return local(op.a) && local(op.b) && op.a != op.b;
    }
    return false;
}

inline int popcount32(uint32_t v) {
    int n = 0;
    for (; v; v &= v - 1) n++;
    return n;
}

ZC_HD bool is_1q(uint32_t kind) { return kind == MOP_U1 || kind == MOP_R1 || kind == MOP_RT; }

// The register group starting at one-qubit op o: three rotations on distinct
// bits (max_group two, the kernel's), else up to max_group one-qubit ops on
// distinct bits. Returns its size; *rot3 tells the first kind.
ZC_HD int group_at(const OpHead *ops, int o, int nops, int max_group, bool *rot3) {
    *rot3 = false;
    if (max_group == 2 && o + 2 < nops && ops[o].kind == MOP_RT && ops[o + 1].kind == MOP_RT &&
        ops[o + 2].kind == MOP_RT && ops[o].a != ops[o + 1].a && ops[o].a != ops[o + 2].a &&
        ops[o + 1].a != ops[o + 2].a) {
        *rot3 = true;
        return 3;
    }
    int g = 1;
    while (g < max_group && o + g < nops && is_1q(ops[o + g].kind)) {
        bool distinct = true;
        for (int h = 0; h < g; h++) distinct &= ops[o + h].a != ops[o + g].a;
        if (!distinct) break;
        g++;
    }
    return g;
}

// Register passes of double-float sweeps, resolved once per job.
//
// A pass is a register group (one to three one-qubit ops on distinct tile
// bits, as group_at forms them) together with the table diagonal right
// before it and, before that, a block of CX ops whose targets are all group
// bits. The diagonal scales each element before the gates, exactly as its
// own pass would. A CX moves data only within a group whose bits hold its
// target, so the CX block becomes the load permutation: logical element y
// (group coordinates; the other bits v fixed) is read from
// pi_1(pi_2(...pi_n(y))), pi_i flipping the target where the control is
// set. Over GF(2) that is y -> M y + sum_i ctl_i(v) w_i: controls among the
// group bits make M, controls outside them (local bits of v, or outer qubits
// fixed per tile) add the translations w_i. The host derives all of it per
// job (encode_job); per tile a pass reads a few shared words.
// Diagonals over eight qubits keep their own trip over the tile (25-qubit QFT
// 9.5 ms; 9.7 with those of up to twelve in passes, whose index bits then cost
// more than the trip).
struct GroupInfo {
    uint8_t G, rot3, skip, first;  // G = 0: no pass starts at this op
    uint8_t nloc, nout, ntr, has_dk;
    uint8_t sorted[3];             // group bits ascending (zero insertion)
    uint8_t tb[3];                 // table bit of each group coordinate (0xff: not in the support)
    uint8_t loc[8], locb[8];       // support bits outside the group -> table bit
    uint8_t outq[8], outb[8];      // outer support qubits -> table bit
    uint8_t trc[4];                // translation controls: local bit, or 0x80 | outer qubit
    uint16_t gm[3];                // slot pattern of group coordinate g (1 << bit)
    uint16_t pm[3];                // load pattern of coordinate g (column g of M, as slots)
    uint16_t trw[4];               // translation patterns
    uint16_t fmask;                // store pattern of the flipped coordinates
    uint16_t so_step, lo_step, jb_step;  // for a thread's second group (set by encode_job)
    uint32_t tab_off;
};

// Walk the ops the way apply_ops will and describe each pass. The kernel's jobs
// have CX blocks folded (fold) and groups of two (max_group); the host check of
// the pass logic also tries single gates and unfolded blocks. *fuse_in /
// *fuse_out: the job starts / ends with a pass, which then also converts the
// tile between f64 and double-float in registers.
inline void plan_passes(const OpHead *ops, int nops, uint32_t tile_log2, bool fold, int max_group, GroupInfo *gi,
                        uint32_t *bad, int *fuse_in, int *fuse_out) {
    for (int i = 0; i < nops; i++) gi[i].G = 0;
    *fuse_out = 0;
    int o = 0;
    while (o < nops) {
        const OpHead &op = ops[o];
        int first = -1, jdk = -1, cx0 = -1, ncx = 0;
        if (fold && op.kind == MOP_CX) {
            int j = o;
            bool ok = true;
            while (j < nops && ops[j].kind == MOP_CX && j - o < kMaxFoldCx) {
                ok &= !(ops[j].b & kOuterFlag);
                j++;
            }
            const bool dk = j < nops && ops[j].kind == MOP_DK && ops[j].k <= 8;
            const int g0 = dk ? j + 1 : j;
            if (ok && g0 < nops && is_1q(ops[g0].kind)) {
                bool rot3;
                const int g = group_at(ops, g0, nops, max_group, &rot3);
                for (int i = o; i < j; i++) {
                    bool hit = false;
                    for (int h = 0; h < g; h++) hit |= ops[g0 + h].a == ops[i].b;
                    ok &= hit;
                }
                if (ok) {
                    first = g0;
                    jdk = dk ? j : -1;
                    cx0 = o;
                    ncx = j - o;
                }
            }
        } else if (op.kind == MOP_DK && op.k <= 8 && o + 1 < nops && is_1q(ops[o + 1].kind)) {
            first = o + 1;
            jdk = o;
        } else if (is_1q(op.kind)) {
            first = o;
        }
        if (first < 0) {
            o++;
            continue;
        }
        bool rot3;
        const int G = group_at(ops, first, nops, max_group, &rot3);
        GroupInfo &q = gi[o];
        uint32_t bits[3] = {0, 0, 0};
        bool in_tile = true;
        for (int g = 0; g < G; g++) {
            bits[g] = ops[first + g].a;
            in_tile &= bits[g] < tile_log2;
        }
        if (!in_tile) {  // not a planned sweep: encode_job refuses the job
            *bad = 0x80000000u | (uint32_t)o;
            o++;
            continue;
        }
        q.G = (uint8_t)G;
        q.rot3 = rot3;
        q.first = (uint8_t)first;
        q.skip = (uint8_t)(first + G - o);
        q.fmask = 0;
        for (int g = 0; g < G; g++) {
            q.gm[g] = q.pm[g] = (uint16_t)(1u << bits[g]);
            if (ops[first + g].kind == MOP_RT && ops[first + g].b) q.fmask |= (uint16_t)(1u << bits[g]);
        }
        uint32_t srt[3] = {bits[0], bits[1], bits[2]};
        for (int a = 1; a < G; a++)
            for (int b = a; b > 0 && srt[b] < srt[b - 1]; b--) {
                const uint32_t x = srt[b];
                srt[b] = srt[b - 1];
                srt[b - 1] = x;
            }
        for (int g = 0; g < 3; g++) q.sorted[g] = (uint8_t)srt[g];
        q.has_dk = jdk >= 0;
        q.nloc = q.nout = 0;
        for (int g = 0; g < 3; g++) q.tb[g] = 0xff;
        if (jdk >= 0) {
            const OpHead &d = ops[jdk];
            q.tab_off = (uint32_t)d.table;
            for (uint32_t b = 0; b < d.k; b++) {
                const uint32_t l = d.loc[b];
                if (l & kOuterFlag) {
                    q.outq[q.nout] = (uint8_t)(l & ~kOuterFlag);
                    q.outb[q.nout++] = (uint8_t)b;
                    continue;
                }
                int hit = -1;
                for (int g = 0; g < G; g++)
                    if (bits[g] == l) hit = g;
                if (hit >= 0) {
                    q.tb[hit] = (uint8_t)b;
                } else {
                    q.loc[q.nloc] = (uint8_t)l;
                    q.locb[q.nloc++] = (uint8_t)b;
                }
            }
        }
        // CX block as an affine map over the group coordinates, composed
        // from the last CX (applied to y first) to the first
        q.ntr = 0;
        if (ncx > 0) {
            uint32_t col[3] = {1u, 2u, 4u}, trv[kMaxFoldCx];
            uint8_t trc[kMaxFoldCx];
            int ntr = 0;
            for (int i = ncx - 1; i >= 0; i--) {
                const OpHead &x = ops[cx0 + i];
                int tau = 0, kap = -1;
                for (int g = 0; g < G; g++) {
                    if (bits[g] == x.b) tau = g;
                    if (!(x.a & kOuterFlag) && bits[g] == x.a) kap = g;
                }
                if (kap >= 0) {  // y_tau ^= y_kap
                    for (int g = 0; g < G; g++)
                        if ((col[g] >> kap) & 1u) col[g] ^= 1u << tau;
                    for (int t = 0; t < ntr; t++)
                        if ((trv[t] >> kap) & 1u) trv[t] ^= 1u << tau;
                } else {  // y_tau ^= (control outside the group)
                    trc[ntr] = x.a & kOuterFlag ? (uint8_t)(0x80u | (x.a & ~kOuterFlag)) : (uint8_t)x.a;
                    trv[ntr++] = 1u << tau;
                }
            }
            auto pattern = [&](uint32_t y) {
                uint32_t w = 0;
                for (int g = 0; g < G; g++)
                    if ((y >> g) & 1u) w |= 1u << bits[g];
                return (uint16_t)w;
            };
            for (int g = 0; g < G; g++) q.pm[g] = pattern(col[g]);
            q.ntr = (uint8_t)ntr;
            for (int t = 0; t < ntr; t++) {
                q.trc[t] = trc[t];
                q.trw[t] = pattern(trv[t]);
            }
        }
        o += q.skip;
        *fuse_out = o == nops;
    }
    *fuse_in = nops > 0 && gi[0].G != 0;
}

// Register passes of f32 sweeps. A pass is a run of consecutive ops whose
// gates and CX targets lie on at most kRegBits tile bits: a thread holds the
// 2^kRegBits elements those bits span and applies the ops in order, each
// element rounded as the ops one by one do. Diagonals join on any support, a
// CX control may lie anywhere. A run with fewer bits is padded with high tile
// bits (low ones would make the lanes of a warp collide in the banks). A lone
// CX stays a permutation pass, which touches half the tile.
constexpr int kRegBits = 4;

struct RegOp {
    uint8_t n;               // ops of the pass that starts here (0: none does)
    uint8_t g;               // the gate's (CX target's) coordinate
    uint8_t c;               // D1 / CX: the coordinate that selects (0xff: not a group bit)
    uint8_t pad;
    uint8_t sorted[4];       // the pass's bits, ascending; coordinate g is sorted[g]
    uint16_t tm[4];          // DK: table index bit of each coordinate (0: not in the support)
};
static_assert(sizeof(RegOp) == 16, "RegOps are copied in 16-byte pieces");

inline void plan_reg_passes(const OpHead *ops, int nops, uint32_t tile_log2, RegOp *out) {
    for (int i = 0; i < nops; i++) out[i] = RegOp{};
    if (tile_log2 < (uint32_t)kRegBits) return;
    for (int o = 0; o < nops;) {
        uint32_t set = 0;
        int n = 0;
        bool arith = false;
        for (; o + n < nops; n++) {
            const OpHead &op = ops[o + n];
            uint32_t add = 0;
            if (op.kind == MOP_U1 || op.kind == MOP_CX) {
                const uint32_t bit = op.kind == MOP_U1 ? op.a : op.b;
                if (bit >= tile_log2) break;  // (encode_job refuses such an op)
                add = 1u << bit;
            } else if (op.kind != MOP_D1 && op.kind != MOP_DK) {
                break;
            }
            if (popcount32(set | add) > kRegBits) break;
            set |= add;
            arith |= op.kind != MOP_CX;
        }
        if (n == 0 || (n == 1 && !arith)) {
            o++;
            continue;
        }
        for (uint32_t b = tile_log2; b-- > 0 && popcount32(set) < kRegBits;) set |= 1u << b;
        uint8_t bits[kRegBits];
        int cnt = 0;
        for (uint32_t b = 0; b < tile_log2; b++)
            if ((set >> b) & 1u) bits[cnt++] = (uint8_t)b;
        auto coord = [&](uint32_t loc) {  // outer locations match no bit
            for (int g = 0; g < kRegBits; g++)
                if (bits[g] == loc) return (uint8_t)g;
            return (uint8_t)0xff;
        };
        out[o].n = (uint8_t)n;
        for (int k = 0; k < n; k++) {
            const OpHead &op = ops[o + k];
            RegOp &r = out[o + k];
            for (int g = 0; g < kRegBits; g++) r.sorted[g] = bits[g];
            r.g = coord(op.kind == MOP_CX ? op.b : op.a);
            r.c = coord(op.a);
            if (op.kind == MOP_DK)
                for (uint32_t b = 0; b < op.k; b++) {
                    const uint8_t g = coord(op.loc[b]);
                    if (g != 0xff) r.tm[g] = (uint16_t)(1u << b);
                }
        }
        o += n;
    }
}

}  // namespace zc
