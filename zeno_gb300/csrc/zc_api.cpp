// C ABI of the backend (include/zeno_cuda.h): state lifecycle, argument
// validation, op dispatch onto the gate kernels, reductions, the sampler's
// host half, and HBM capacity planning.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "zc_internal.h"
#include "zc_rng.h"
#include "zc_sweep.h"

namespace zc {

static thread_local std::string g_err;

const char *const kKernelNames[K_NKINDS] = {"1q",         "kq",         "diag1",       "diagk",    "cx",
                                            "swap",       "sweep",      "chunk_sums",  "serial_sum", "sample_scan",
                                            "collapse",   "reset",      "trajectories", "tc_block"};

ProfScope::ProfScope(zc_state *s, int kind, double bytes) : st(s) {
    if (!st || !st->prof) return;
    cudaEvent_t ev[2];
    for (int i = 0; i < 2; i++) {
        if (!st->prof_pool.empty()) {
            ev[i] = st->prof_pool.back();
            st->prof_pool.pop_back();
        } else if (cudaEventCreate(&ev[i]) != cudaSuccess) {
            return;
        }
    }
    cudaEventRecord(ev[0], st->stream);
    st->prof_recs.push_back(ProfRec{kind, bytes, ev[0], ev[1]});
    idx = (long)st->prof_recs.size() - 1;
}

ProfScope::~ProfScope() {
    if (idx >= 0) cudaEventRecord(st->prof_recs[idx].b, st->stream);
}

int fail(int code, const std::string &msg) {
    g_err = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char *where) {
    g_err = std::string("CUDA error in ") + where + ": " + cudaGetErrorString(e);
    return ZC_ERR_CUDA;
}

static std::string human_bytes(double b) {
    const char *units[] = {"B", "KiB", "MiB", "GiB", "TiB"};
    int u = 0;
    while (b >= 1024.0 && u < 4) {
        b /= 1024.0;
        u++;
    }
    char buf[64];
    if (u == 0)
        snprintf(buf, sizeof buf, "%.0f B", b);
    else
        snprintf(buf, sizeof buf, "%.1f %s", b, units[u]);
    return buf;
}

static constexpr size_t kArenaBytes = 32u << 20;

// Copy `bytes` into the device parameter ring and return its device address.
int arena_put(zc_state *st, const void *src, size_t bytes, const void **dev) {
    Arena &a = st->arena;
    const size_t need = (bytes + 255) & ~(size_t)255;
    if (need > a.cap) return fail(ZC_ERR_INVALID, "op table larger than the parameter arena");
    if (a.head + need > a.cap) {
        ZC_CUDA(cudaStreamSynchronize(st->stream));
        a.head = 0;
    }
    memcpy(a.host + a.head, src, bytes);
    ZC_CUDA(cudaMemcpyAsync(a.dev + a.head, a.host + a.head, bytes, cudaMemcpyHostToDevice, st->stream));
    *dev = a.dev + a.head;
    a.head += need;
    return ZC_OK;
}

// Stage a complex table (interleaved c64) as split T arrays [re..., im...].
static int stage_table(zc_state *st, const double *c64, size_t count, const void **dev) {
    if (st->prec == 64) {
        std::vector<double> t(2 * count);
        for (size_t i = 0; i < count; i++) {
            t[i] = c64[2 * i];
            t[count + i] = c64[2 * i + 1];
        }
        return arena_put(st, t.data(), t.size() * sizeof(double), dev);
    }
    std::vector<float> t(2 * count);
    for (size_t i = 0; i < count; i++) {
        t[i] = (float)c64[2 * i];
        t[count + i] = (float)c64[2 * i + 1];
    }
    return arena_put(st, t.data(), t.size() * sizeof(float), dev);
}

static int check_support(const zc_state *st, const uint32_t *qs, uint32_t k, uint32_t kmax, const char *what) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    if (k < 1 || k > kmax) return fail(ZC_ERR_INVALID, std::string(what) + ": support size out of range");
    if (!qs) return fail(ZC_ERR_INVALID, std::string(what) + ": null qubit list");
    for (uint32_t i = 0; i < k; i++) {
        if (qs[i] >= st->n) return fail(ZC_ERR_INVALID, std::string(what) + ": qubit out of range");
        if (i && qs[i] <= qs[i - 1])
            return fail(ZC_ERR_INVALID, std::string(what) + ": qubits must be sorted and distinct");
    }
    return ZC_OK;
}

static inline bool exact(const zc_state *st) { return (st->flags & ZC_FLAG_FAST) == 0; }
// The arithmetic of the ops being launched (see few_in_exact).
static inline bool exact_ops(const zc_state *st) { return exact(st) || st->exact_flush; }


void touch_pages(void *p, size_t bytes) {
    static const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    volatile char *c = (volatile char *)p;
    for (size_t b = 0; b < bytes; b += b ? page : page - (uintptr_t)p % page) c[b] = 0;
}

int sync_status(zc_state *st) {
    ZC_CUDA(cudaMemcpyAsync(st->h_scalar, st->d_scalar, kStatusErr + sizeof(int), cudaMemcpyDeviceToHost,
                            st->stream));
    ZC_CUDA(cudaStreamSynchronize(st->stream));
    const int *h = (const int *)((const char *)st->h_scalar + kStatusErr);
    return h[0] ? check_device_error(st) : ZC_OK;  // a kernel that gave up leaves a wrong state behind
}

static int sync_read_scalar(zc_state *st, double *out) {
    const int rc = sync_status(st);
    *out = *st->h_scalar;
    return rc;
}

static int grow(void **p, size_t *cap, size_t need) {
    if (need <= *cap) return ZC_OK;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    ZC_CUDA(cudaMalloc(p, need));
    *cap = need;
    return ZC_OK;
}


// ------------------------------------------------------------------ scheduling

static constexpr size_t kQueueWindow = 2048;  // ops examined per sweep plan
static constexpr size_t kQueueFlushAt = 8192; // queue length that forces a flush
static constexpr uint32_t kMinSweepQubits = 3;

int launch_single(zc_state *st, const QOp &op) {
    const bool ex = exact_ops(st);
    switch (op.kind) {
        case Q_UNITARY: {
            if (op.k == 1) return launch_1q(st, op.qs[0], op.data.data(), ex);
            if (op.k >= 3 && st->prec == 32 && (st->flags & ZC_FLAG_TENSOR))
                return launch_block_tc(st, op.qs, op.k, op.data.data());
            if (op.k <= kMaxRegUnitary && !(op.k == 4 && ex && st->prec == 64 && st->n < kStagedK4Qubits))
                return launch_kq_small(st, op.qs, op.k, op.data.data(), ex);
            const void *dev = nullptr;
            if (st->prec == 64 && !ex) {  // fast f64: double-float on the FP32 pipe
                const size_t cnt = (size_t)1 << (2 * op.k);
                std::vector<float> t(4 * cnt);
                for (size_t i = 0; i < cnt; i++) {
                    for (int part = 0; part < 2; part++) {  // re, im: hi = nearest float, lo = the rest
                        const double x = op.data[2 * i + part];
                        const float hi = (float)x;
                        t[4 * i + 2 * part] = hi;
                        t[4 * i + 2 * part + 1] = (float)(x - (double)hi);
                    }
                }
                int rc = arena_put(st, t.data(), t.size() * sizeof(float), &dev);
                if (rc) return rc;
                return launch_kq_df(st, op.qs, op.k, dev);
            }
            int rc = stage_table(st, op.data.data(), (size_t)1 << (2 * op.k), &dev);
            if (rc) return rc;
            return launch_kq(st, op.qs, op.k, dev, ex);
        }
        case Q_DIAG: {
            if (op.k == 1) return launch_diag1(st, op.qs[0], op.data.data(), ex);
            const void *dev = nullptr;
            int rc = stage_table(st, op.data.data(), (size_t)1 << op.k, &dev);
            if (rc) return rc;
            return launch_diagk(st, op.qs, op.k, dev, ex);
        }
        case Q_CX:
            return launch_cx(st, op.a, op.b);
        default:
            return launch_swap(st, op.a, op.b);
    }
}

// Qubits that must be local for `op` to run inside a sweep.
static uint64_t need_mask(const QOp &op) {
    switch (op.kind) {
        case Q_UNITARY: return 1ull << op.qs[0];
        case Q_DIAG: return 0;
        case Q_CX: return 1ull << op.b;
        default: return (1ull << op.a) | (1ull << op.b);
    }
}

static bool sweepable(const QOp &op) { return !(op.kind == Q_UNITARY && op.k > 1); }

struct SweepShape {
    uint32_t L, Hcap;
};

// How many high qubits a tile takes. A sweep costs ~15 us of planning, copy and
// launch, so a small state wants tiles that hold many of its qubits (fewer
// sweeps), against enough tiles for the SMs. Measured per whole zc_run
// (depth-12 u3 + matching CX; f32: gate mix), us:
//   exact f64, bound by each SM's FP64 pipe: 2^8 amplitudes per tile up to 15
//   qubits (12q: 718 with 2^8, 1322 with 2^11), 2^9 for 16-17, 2^10 for 18-21
//   (20q: 5529, 2^11 5699), whole tiles beyond (22q: 6600)
//   double-float: about half the qubits plus two, at least 2^8 (10q 355, one
//   launch per op 842; 16q 544 with 2^10, 918 with 2^7; 20q 1080 with 2^12)
//   f32: up to 13 qubits the state is one tile (10q 155, one launch per op
//   408); larger states keep at least two tiles per SM
static SweepShape shape_for(const zc_state *st) {
    const uint32_t n = st->n, L = std::min<uint32_t>(n, st->prec == 64 ? 5 : 6);  // 256-byte rows
    const uint32_t Tmax = st->prec == 64 ? 12 : 13;                                // 64 KiB per tile buffer
    uint32_t Hcap = std::min<uint32_t>(Tmax - L, n - L);
    if (st->sweep_high) return SweepShape{L, std::min<uint32_t>(Hcap, st->sweep_high)};  // tuned
    uint32_t T = Tmax;
    if (st->prec == 64 && exact_ops(st)) {
        T = n <= 15 ? 8 : n <= 17 ? 9 : n <= 21 ? 10 : Tmax;
    } else if (st->prec == 64) {
        T = std::max<uint32_t>(8, n / 2 + 2);
    } else if (n >= kSmallStateQubits) {
        uint32_t tiles_log2 = 0;
        while ((1u << tiles_log2) < (uint32_t)(2 * st->num_sms)) tiles_log2++;
        T = n - std::min(tiles_log2, n - L);
    }
    return SweepShape{L, std::min(Hcap, std::max(T, L) - L)};
}

// Whether ops keep program order. Exact mode does (reordering two gates
// changes the rounding); so do small f32 states, whose results stay those of
// one launch per op.
static bool program_order(const zc_state *st) {
    return exact_ops(st) || (st->prec == 32 && st->n < kSmallStateQubits);
}

// A few queued ops on a small state. A sweep costs ~20 us of planning, copy and
// latency before its first op, a double-float one ~40. Measured from a caller's
// first op to the end, us:
//   f32, 8 qubits, in a sweep / one by one: 2 ops 34/24, 3 39/32, 4 42/44, 6
//   51/57: fewer than four go one by one, the same bits
//   fast f64, 8 qubits, in double-float / in exact arithmetic: 2 ops 41/33, 3
//   59/38, 6 74/50, 10 92/66; through zc_run (whole calls) 4 167/153, 7 168/169,
//   8 174/195, at 13 qubits 4 176/170, 6 181/183, 8 182/209: two to seven run
//   in exact arithmetic, which is also the closer one (6 ops at 8 qubits: 5e-17
//   off, 1e-15 in a double-float sweep). One by one in double-float 2 ops take
//   32 but are five times further off than in a sweep: each launch converts to
//   pairs and back. Dense blocks, whose exact sums take twice as long, keep
//   their own way.
static constexpr size_t kFewF32 = 4, kFewF64 = 8;
static bool few_ops(const zc_state *st, size_t few) {
    return hides_queue(st) && st->queue.size() < few;
}
static bool few_one_by_one(const zc_state *st) { return st->prec == 32 && few_ops(st, kFewF32); }
static bool few_in_exact(const zc_state *st) {
    if (st->prec == 32 || exact(st) || !few_ops(st, kFewF64) || st->queue.size() < 2) return false;
    for (size_t i = 0; i < st->queue.size(); i++)
        if (!sweepable(st->queue[i])) return false;
    return true;
}

static uint32_t loc_of(uint32_t q, uint32_t L, const std::vector<uint32_t> &highs) {
    if (q < L) return q;
    for (size_t j = 0; j < highs.size(); j++)
        if (highs[j] == q) return L + (uint32_t)j;
    return kOuterFlag | q;
}

// Choose the ops of one sweep from the queue front (see the scheduling
// rules above). Fills `plan` and returns how many ops it took; 0 or 1 means
// the front op should simply run on its own.
size_t plan_sweep(uint32_t n, int prec, bool ex, uint32_t L, uint32_t Hcap, const std::vector<QOp> &q,
                  SweepPlan *plan, size_t head, uint64_t touch_all) {
    const uint64_t low_mask = L >= 64 ? ~0ull : ((1ull << L) - 1);
    uint64_t blocked = 0, highs_mask = 0;
    uint32_t nhigh = 0;
    bool arith_deferred = false;
    std::vector<size_t> &taken = plan->taken;
    taken.clear();
    const size_t window = head + std::min(q.size() - head, kQueueWindow);
    const uint64_t qubits = touch_all & (n >= 64 ? ~0ull : (1ull << n) - 1);
    // Under double-float lowering a diagonal joins the pending tables and
    // becomes a micro-op only when flushed, so it does not count against the
    // micro-op budget here (the lowered count is checked below).
    const bool df_lowering = !ex && prec == 64;
    size_t counted = 0;
    // once every qubit is blocked no later op can join (walking the rest of the
    // window regardless cost 5 us per lone op)
    for (size_t i = head; i < window && counted < (size_t)kMaxMicroOps &&
                          taken.size() < 4 * (size_t)kMaxMicroOps && (blocked & qubits) != qubits;
         i++) {
        const QOp &op = q[i];
        const uint64_t touch = touch_mask(op);
        const bool arith = op.kind == Q_UNITARY || op.kind == Q_DIAG;
        bool defer = (touch & blocked) != 0 || (ex && arith && arith_deferred) || !sweepable(op);
        uint64_t need = 0;
        if (!defer) {
            need = need_mask(op) & ~low_mask & ~highs_mask;
            if (nhigh + (uint32_t)__builtin_popcountll(need) > Hcap) defer = true;
        }
        if (defer) {
            blocked |= touch;
            arith_deferred |= arith;
            continue;
        }
        highs_mask |= need;
        nhigh += (uint32_t)__builtin_popcountll(need);
        taken.push_back(i);
        counted += !(df_lowering && op.kind == Q_DIAG);
    }
    if (taken.size() <= 1) return taken.size();
    // pad the tile with further high qubits up to the cap (no effect on results)
    for (uint32_t b = L; b < n && nhigh < Hcap; b++)
        if (!((highs_mask >> b) & 1)) {
            highs_mask |= 1ull << b;
            nhigh++;
        }
    std::vector<uint32_t> highs;
    for (uint32_t b = 0; b < n; b++)
        if ((highs_mask >> b) & 1) highs.push_back(b);
    SweepGeom &g = plan->g;
    g = SweepGeom{};
    g.n = n;
    g.L = L;
    g.H = (uint32_t)highs.size();
    for (size_t j = 0; j < highs.size(); j++) g.hpos[j] = highs[j];
    g.ntiles = 1ull << (n - g.L - g.H);
    // Order of the micro-ops. Exact mode keeps program order (reordering two
    // gates changes the rounding). Fast mode lets ops on disjoint qubits
    // commute: one-qubit ops on distinct qubits are emitted back to back, in
    // runs (three for the rotations of lowered f64 sweeps, their register group;
    // else two: an f32 pass takes four tile bits in whatever order, and another
    // run length would round f32 states differently).
    const size_t run_cap = prec == 32 ? 2 : (prec == 64 && !df_lowering ? 2 : 3);
    const bool df = df_lowering;
    std::vector<LoweredOp> low;
    for (;;) {
    std::vector<size_t> order(taken.size());
    for (size_t t = 0; t < taken.size(); t++) order[t] = t;
    if (!ex) {
        const size_t m = taken.size();
        std::vector<char> done(m, 0);
        std::vector<uint64_t> touch(m);
        for (size_t i = 0; i < m; i++) touch[i] = touch_mask(q[taken[i]]);
        auto is1q = [&](size_t i) { return q[taken[i]].kind == Q_UNITARY && q[taken[i]].k == 1; };
        const uint64_t all = n >= 64 ? ~0ull : ((1ull << n) - 1);
        order.clear();
        uint64_t cx_targets = 0;  // targets of the CX ops since the last run
        size_t first = 0;         // ops before it are emitted
        while (order.size() < m) {
            while (done[first]) first++;
            // ready one-qubit ops on distinct qubits, program order; those on
            // targets of the CX ops just emitted first (the kernel folds a CX
            // into the register group that holds its target). An op is ready
            // when no op before it that is still to come touches its qubits.
            std::vector<size_t> run;
            uint64_t used = 0;
            size_t other = m;  // the first ready op of another kind
            for (int pass = 0; pass < 2 && run.size() < run_cap; pass++) {
                uint64_t ahead = 0;
                for (size_t i = first; i < m && run.size() < run_cap && ahead != all; i++) {
                    if (done[i]) continue;
                    const bool ready = !(touch[i] & ahead);
                    ahead |= touch[i];
                    if (!ready) continue;
                    if (!is1q(i)) {
                        other = std::min(other, i);
                        continue;
                    }
                    const uint32_t qb = q[taken[i]].qs[0];
                    if ((used >> qb) & 1) continue;
                    if (pass == 0 && !((cx_targets >> qb) & 1)) continue;
                    run.push_back(i);
                    used |= 1ull << qb;
                }
            }
            std::sort(run.begin(), run.end());
            // a full run goes out at once; otherwise a ready op of another
            // kind goes first (it can make more one-qubit ops ready), and a
            // short run only when nothing else is ready
            if (run.size() < run_cap && other < m) {
                done[other] = 1;
                order.push_back(other);
                if (q[taken[other]].kind == Q_CX) cx_targets |= 1ull << q[taken[other]].b;
                continue;
            }
            for (size_t i : run) {
                done[i] = 1;
                order.push_back(i);
            }
            cx_targets = 0;
        }
    }
    // Lowering: double-float sweeps of f64 states rewrite one-qubit gates as
    // diagonal * real * diagonal and merge the diagonals; other policies
    // encode the ops as they are.
    low.clear();
    plan->carry.clear();
    if (df) {
        std::vector<const QOp *> seq;
        for (size_t t : order) seq.push_back(&q[taken[t]]);
        // a sweep with no sweep to follow at once (the queue ends or a dense block
        // is next) applies its pending diagonals itself, if they fit: carried,
        // they would be a launch of their own
        size_t next = head;
        while (next - head < taken.size() && taken[next - head] == next) next++;
        const bool last = next == q.size() || !sweepable(q[next]);
        lower_df(seq, 2, &low, last ? nullptr : &plan->carry);
        if (last && low.size() > (size_t)kMaxMicroOps) {
            low.clear();
            lower_df(seq, 2, &low, &plan->carry);
        }
    } else {
        for (size_t t : order) {
            const QOp &op = q[taken[t]];
            LoweredOp o{};
            if (op.kind == Q_UNITARY) {
                o.kind = MOP_U1;
                o.a = op.qs[0];
                for (int i = 0; i < 8; i++) o.m[i] = op.data[i];
            } else if (op.kind == Q_DIAG) {
                o.kind = MOP_DK;
                o.sup.assign(op.qs, op.qs + op.k);
                o.tab = op.data;
            } else {
                o.kind = op.kind == Q_CX ? MOP_CX : MOP_SWAP;
                o.a = op.a;
                o.b = op.b;
            }
            low.push_back(std::move(o));
        }
    }
    if (low.size() <= (size_t)kMaxMicroOps) break;
    // lowering added table ops: take fewer queue ops (dropping the last
    // taken ops never breaks an ordering constraint), first in proportion
    // (lowering again costs more than an op in the next sweep), then singly
    const size_t fit = taken.size() * (size_t)kMaxMicroOps / low.size();
    taken.resize(std::min(fit, taken.size() - 1));
    if (taken.size() <= 1) {
        taken.assign(1, head);
        plan->carry.clear();
        return taken.size();
    }
    }
    std::vector<MicroOp> &mops = plan->mops;
    std::vector<char> &tables = plan->tables;
    mops.assign(low.size(), MicroOp{});
    tables.clear();
    const size_t es = prec / 8;
    for (size_t t = 0; t < low.size(); t++) {
        const LoweredOp &op = low[t];
        MicroOp &m = mops[t];
        if (op.kind == MOP_U1 || op.kind == MOP_R1 || op.kind == MOP_RT) {
            m.kind = op.kind;
            m.a = loc_of(op.a, g.L, highs);
            if (op.kind == MOP_RT) m.b = op.b;  // form
            for (int i = 0; i < 8; i++) m.m[i] = op.m[i];
        } else if (op.kind == MOP_DK && op.sup.size() == 1 && !df) {  // double-float: tables ride in groups
            m.kind = MOP_D1;
            m.a = loc_of(op.sup[0], g.L, highs);
            for (int i = 0; i < 4; i++) m.m[i] = op.tab[i];
        } else if (op.kind == MOP_DK) {
            m.kind = MOP_DK;
            m.k = (uint32_t)op.sup.size();
            for (uint32_t b = 0; b < m.k; b++) m.loc[b] = loc_of(op.sup[b], g.L, highs);
            const size_t dim = (size_t)1 << m.k;
            size_t off = (tables.size() + 15) & ~(size_t)15;
            tables.resize(off + 2 * dim * es);
            for (size_t j = 0; j < dim; j++) {
                const double xr = op.tab[2 * j], xi = op.tab[2 * j + 1];
                if (df) {  // (re hi, re lo, im hi, im lo)
                    float *e = (float *)(tables.data() + off) + 4 * j;
                    e[0] = (float)xr;
                    e[1] = (float)(xr - (double)e[0]);
                    e[2] = (float)xi;
                    e[3] = (float)(xi - (double)e[2]);
                } else if (es == 8) {  // (re, im) pairs: one 16-byte load per entry
                    ((double *)(tables.data() + off))[2 * j] = xr;
                    ((double *)(tables.data() + off))[2 * j + 1] = xi;
                } else {
                    ((float *)(tables.data() + off))[2 * j] = (float)xr;
                    ((float *)(tables.data() + off))[2 * j + 1] = (float)xi;
                }
            }
            m.table = off;
        } else {
            m.kind = op.kind;
            m.a = loc_of(op.a, g.L, highs);
            m.b = loc_of(op.b, g.L, highs);
        }
    }
    return taken.size();
}

// The ops that stay move up against those behind the plan's reach, so the cost
// is that of the plan's own span. The carried diagonals act after every op the
// sweep took and touch only qubits those ops touched; no op deferred ahead of
// them touches those qubits, so the queue front is their place in program order.
void consume_plan(std::vector<QOp> &q, SweepPlan &plan, size_t *head) {
    size_t from = head ? *head : 0;
    if (!plan.taken.empty()) {
        size_t w = plan.taken.back() + 1, ti = plan.taken.size();
        for (size_t i = w; i-- > from;) {
            if (ti && plan.taken[ti - 1] == i) {
                ti--;
                std::vector<double>().swap(q[i].data);
                continue;
            }
            if (--w != i) q[w] = std::move(q[i]);
        }
        from = w;
    }
    if (plan.carry.size() > from) {  // (a plan carries fewer diagonals than it took ops)
        q.insert(q.begin() + (long)from, plan.carry.size() - from, QOp{});
        from = plan.carry.size();
    }
    while (!plan.carry.empty()) {
        q[--from] = std::move(plan.carry.back());
        plan.carry.pop_back();
    }
    if (head) *head = from;
    else q.erase(q.begin(), q.begin() + (long)from);
}

// Ops of a fast f64 state that read and leave packed double-float pairs.
static bool takes_pairs(const QOp &op) { return sweepable(op) || (op.kind == Q_UNITARY && op.k <= kMaxRegUnitary); }
static bool sweeps_enabled(const zc_state *st);

// Before any kernel other than a sweep: a state that double-float sweeps
// left as packed float pairs goes back to f64.
static int settle_form(zc_state *st) {
    if (!st->df_resident) return ZC_OK;
    st->df_resident = false;
    return launch_df_to_f64(st);
}

// Plan and launch one sweep starting at the queue front; takes out what ran.
static int run_one_sweep(zc_state *st) {
    OpQueue &q = st->queue;
    const SweepShape sh = shape_for(st);
    SweepPlan plan;
    if (plan_sweep(st->n, st->prec, program_order(st), sh.L, sh.Hcap, q.ops, &plan, q.head, q.touch) <= 1) {
        // nothing to batch: the per-op kernel is the same work (a permutation
        // moves slots whatever they hold)
        const bool perm = q.front().kind == Q_CX || q.front().kind == Q_SWAP;
        int rc = perm ? ZC_OK : settle_form(st);
        if (rc) return rc;
        rc = launch_single(st, q.front());
        q.pop();
        return rc;
    }
    std::vector<char> blob;
    int rc = encode_job(st->prec, exact_ops(st), plan, &blob);
    if (rc) return rc;
    const size_t tab_off = (blob.size() + 255) & ~(size_t)255;
    blob.resize(tab_off + plan.tables.size());
    if (!plan.tables.empty()) memcpy(blob.data() + tab_off, plan.tables.data(), plan.tables.size());
    const void *dev = nullptr;
    rc = arena_put(st, blob.data(), blob.size(), &dev);
    if (rc) return rc;
    consume_plan(q.ops, plan, &q.head);
    // Fast f64: consecutive sweeps of one flush hand the state over as
    // (hi, lo) float pairs, also to and from small dense blocks; the last one
    // (nothing that takes pairs queued behind it) rounds it back to f64.
    const bool df = st->prec == 64 && !exact_ops(st);
    const bool out_df = df && !q.empty() && takes_pairs(q.front());
    plan.g.form = (st->df_resident ? kFormInDf : 0u) | (out_df ? kFormOutDf : 0u);
    rc = launch_sweep(st, plan.g, (const char *)dev, (const char *)dev + tab_off, exact_ops(st));
    st->df_resident = out_df;
    for (const MicroOp &m : plan.mops) st->ctr.micro_ops[m.kind & 7]++;
    return rc;
}

static bool sweeps_enabled(const zc_state *st) {
    return !(st->flags & ZC_FLAG_NO_SWEEPS) && st->n >= kMinSweepQubits;
}

// Launch everything queued (program order preserved where results depend on it).
int flush(zc_state *st) {
    int rc = ZC_OK;
    st->exact_flush = few_in_exact(st);
    if (few_one_by_one(st))
        while (!st->queue.empty() && rc == ZC_OK) {
            rc = launch_single(st, st->queue.front());
            st->queue.pop();
        }
    while (!st->queue.empty() && rc == ZC_OK) {
        if (!sweeps_enabled(st) || !sweepable(st->queue.front())) {
            const QOp &op = st->queue.front();
            if (st->prec == 64 && !exact_ops(st) && sweeps_enabled(st) && takes_pairs(op)) {  // a small dense block
                const bool out_df = st->queue.size() > 1 && takes_pairs(st->queue[1]);
                rc = launch_kq_small(st, op.qs, op.k, op.data.data(), false, st->df_resident, out_df);
                st->df_resident = out_df;
            } else {
                rc = settle_form(st);
                if (rc == ZC_OK) rc = launch_single(st, op);
            }
            st->queue.pop();
            continue;
        }
        rc = run_one_sweep(st);
    }
    st->queue.clear();
    st->exact_flush = false;
    const int rc2 = settle_form(st);  // every other entry point sees f64
    return rc ? rc : rc2;
}

// The kernels a queued op of a small state may launch, loaded as it is applied:
// its launch may come inside a call that allocates nothing. Once per device,
// arithmetic and kind of op (2 MB of device memory for the double-float sweeps,
// the other kinds none that shows).
static int load_for(const zc_state *st, const QOp &op) {
    static std::atomic<uint64_t> loaded[64];
    const bool ex = exact(st), tc = op.kind == Q_UNITARY && op.k >= 3 && st->prec == 32 && (st->flags & ZC_FLAG_TENSOR);
    const uint32_t k = sweepable(op) ? 1 : op.k;
    const uint64_t bit = 1ull << ((st->prec == 64) * 32 + ex * 16 + tc * 8 + k);
    std::atomic<uint64_t> &mask = loaded[st->device & 63];
    if (mask.load(std::memory_order_relaxed) & bit) return ZC_OK;
    int rc = tc ? load_tc_kernels(k) : load_op_kernels(st->prec, ex, k);
    if (rc == ZC_OK && k == 1) rc = load_sweep_kernels(st->prec, ex);
    if (rc == ZC_OK && k == 1 && st->prec == 64 && !ex) {  // few_in_exact
        rc = load_op_kernels(64, true, 1);
        if (rc == ZC_OK) rc = load_sweep_kernels(64, true);
    }
    if (rc == ZC_OK) mask.fetch_or(bit, std::memory_order_relaxed);
    return rc;
}

static int enqueue(zc_state *st, QOp &&op) {
    st->ctr.ops++;
    if (!sweeps_enabled(st) || st->stream_out) return launch_single(st, op);
    if (hides_queue(st)) {
        const int rc = load_for(st, op);
        if (rc) return rc;
    }
    // A dense block on a small state ends what can be batched: launching it now
    // lets the device work while the caller goes on (4 qubits, blocks with two ops
    // between them: f32 8.7 -> 5.1 us per op). In fast f64 it stays, so that
    // sweeps and blocks hand float pairs on.
    const bool at_once = hides_queue(st) && !sweepable(op) && (st->prec == 32 || exact(st));
    st->queue.push(std::move(op));
    if (at_once || st->queue.size() >= kQueueFlushAt) return flush(st);
    return ZC_OK;
}

int check_device_error(zc_state *st) {
    int h = 0;
    ZC_CUDA(cudaMemcpyAsync(&h, st->d_err, sizeof(h), cudaMemcpyDeviceToHost, st->stream));
    ZC_CUDA(cudaStreamSynchronize(st->stream));
    if (!h) return ZC_OK;
    cudaMemsetAsync(st->d_err, 0, sizeof(h), st->stream);
    return fail(ZC_ERR_CUDA, "tensor-core block kernel gave up waiting for a copy or an MMA (device wait limit)");
}

// Sampler host half (src/sample.rs:51-62), exactly as the reference orders
// it: serial prefix of the chunk masses, `shots` serial draws scaled by the
// total, ascending sort, and the routing of draws to chunks
// (partition_point(u < cum_before[c])).
void sample_route(const double *sums, size_t nch, uint64_t len, uint64_t shots, uint64_t seed, SampleRoute *r) {
    std::vector<double> cum(nch + 1);
    cum[0] = 0.0;
    for (size_t c = 0; c < nch; c++) cum[c + 1] = cum[c] + sums[c];
    const double total = cum[nch];
    Xoshiro rng(seed);
    r->us.resize(shots);
    for (uint64_t i = 0; i < shots; i++) r->us[i] = rng.f64() * total;
    std::sort(r->us.begin(), r->us.end());
    r->touched.clear();
    size_t prev = std::lower_bound(r->us.begin(), r->us.end(), cum[0]) - r->us.begin();
    for (size_t c = 0; c < nch; c++) {
        const size_t next = std::lower_bound(r->us.begin(), r->us.end(), cum[c + 1]) - r->us.begin();
        if (prev < next) r->touched.push_back(SampleChunk{c, prev, next, cum[c]});
        prev = next;
    }
    r->chunk_len = len < (1ull << kSampleChunkLog2) ? len : (1ull << kSampleChunkLog2);
}

static size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t sample_pass2_bytes(const zc_state *st, const SampleRoute &r) {
    return up256(r.us.size() * sizeof(uint64_t)) + up256(r.us.size() * sizeof(double)) +
           up256(r.touched.size() * sizeof(SampleChunk)) + sample_scan_scratch(r.touched.size(), r.chunk_len, exact(st));
}

// Pass 2, asynchronous. d_work (sample_pass2_bytes(st, r) bytes, 256-aligned)
// holds [indices | draws | touched chunks | rescan scratch]; draws and chunk
// lists small enough travel through the pinned parameter ring, larger ones
// are copied from pageable memory (which waits for the stream).
int sample_launch_pass2(zc_state *st, const SampleRoute &r, char *d_work, uint64_t **d_out) {
    const size_t shots = r.us.size();
    uint64_t *out = (uint64_t *)d_work;
    *d_out = out;
    if (shots == 0) return ZC_OK;
    const size_t out_b = up256(shots * sizeof(uint64_t)), us_b = up256(shots * sizeof(double));
    const size_t cs_b = up256(r.touched.size() * sizeof(SampleChunk));
    const size_t cs_n = r.touched.size() * sizeof(SampleChunk);
    const void *d_us = d_work + out_b, *d_cs = d_work + out_b + us_b;
    int rc = ZC_OK;
    // Through the ring only when both fit in a quarter of it: if the second
    // put wraps, the first began past three quarters, beyond the reach of the
    // second (placed at offset 0), so the kernel reads both intact.
    if (shots * sizeof(double) + cs_n <= st->arena.cap / 4) {
        rc = arena_put(st, r.us.data(), shots * sizeof(double), &d_us);
        if (rc == ZC_OK && cs_n) rc = arena_put(st, r.touched.data(), cs_n, &d_cs);
        if (rc) return rc;
    } else {
        ZC_CUDA(cudaMemcpyAsync((void *)d_us, r.us.data(), shots * sizeof(double), cudaMemcpyHostToDevice, st->stream));
        if (cs_n)
            ZC_CUDA(cudaMemcpyAsync((void *)d_cs, r.touched.data(), cs_n, cudaMemcpyHostToDevice, st->stream));
    }
    ZC_CUDA(cudaMemsetAsync(out, 0, shots * sizeof(uint64_t), st->stream));
    char *scratch = d_work + out_b + us_b + cs_b;
    return launch_sample_scan(st, (const SampleChunk *)d_cs, r.touched.size(), (const double *)d_us, out, r.chunk_len,
                              exact(st), scratch);
}

}  // namespace zc

using namespace zc;

extern "C" {

const char *zc_last_error(void) { return g_err.c_str(); }

uint64_t zc_state_bytes(uint32_t n, int prec) { return (n >= 64 ? 0 : (1ull << n)) * (prec == 32 ? 8u : 16u); }

uint32_t zc_max_qubits(uint64_t budget, int prec) {
    uint32_t n = 0;
    while ((((unsigned __int128)1) << (n + 1)) * (unsigned __int128)(prec == 32 ? 8 : 16) <= budget) {
        n++;
        if (n >= 60) break;
    }
    return n;
}

// physical_ram_bytes (src/mem.rs:9-16) for the device: ZENO_MEM_BYTES
// pretends to be a device of that many bytes, else the device's total HBM.
static int device_memory(uint64_t *bytes) {
    const char *env = getenv("ZENO_MEM_BYTES");
    if (env && *env) {
        char *end = nullptr;
        unsigned long long v = strtoull(env, &end, 10);
        if (end && *end == 0) {
            *bytes = v;
            return ZC_OK;
        }
    }
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemGetInfo");
    *bytes = total_b;
    return ZC_OK;
}

// budget_bytes without an explicit limit (src/mem.rs:104-111).
int zc_device_budget(double fraction, uint64_t *bytes) {
    if (!bytes) return fail(ZC_ERR_INVALID, "null output");
    uint64_t mem = 0;
    const int rc = device_memory(&mem);
    if (rc) return rc;
    *bytes = (uint64_t)((double)mem * fraction);
    return ZC_OK;
}

int zc_device_memory(uint64_t *bytes) {
    if (!bytes) return fail(ZC_ERR_INVALID, "null output");
    return device_memory(bytes);
}

int zc_device_info(zc_device *out) {
    if (!out) return fail(ZC_ERR_INVALID, "null output");
    memset(out, 0, sizeof *out);
    int dev = 0;
    ZC_CUDA(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    ZC_CUDA(cudaGetDeviceProperties(&prop, dev));
    snprintf(out->name, sizeof out->name, "%s", prop.name);
    out->sms = (uint32_t)prop.multiProcessorCount;
    out->cc_major = (uint32_t)prop.major;
    out->cc_minor = (uint32_t)prop.minor;
    size_t free_b = 0, total_b = 0;
    ZC_CUDA(cudaMemGetInfo(&free_b, &total_b));
    out->hbm_bytes = total_b;
    out->free_bytes = free_b;
    out->l2_bytes = (uint64_t)prop.l2CacheSize;
    return ZC_OK;
}

int zc_create(uint32_t n, int prec, zc_state **out) { return zc_create_ex(n, prec, ZC_FLAG_EXACT, out); }

}  // extern "C"

namespace zc {

// mem::plan (src/mem.rs:114-131): refuse a state above the budget, with the
// text of zeno's Error::Memory.
int plan_state(uint32_t n, int prec, uint64_t budget) {
    const uint64_t need = zc_state_bytes(n, prec);
    if (need > budget) {
        char buf[256];
        snprintf(buf, sizeof buf,
                 "state vector for %u qubits at f%d needs %s but the budget is %s (max %u qubits at this "
                 "precision; raise --mem-limit or lower qubits)",
                 n, prec, human_bytes((double)need).c_str(), human_bytes((double)budget).c_str(),
                 zc_max_qubits(budget, prec));
        return fail(ZC_ERR_MEMORY, buf);
    }
    return ZC_OK;
}

}  // namespace zc

extern "C" int zc_create_ex(uint32_t n, int prec, uint32_t flags, zc_state **out) {
    if (!out) return fail(ZC_ERR_INVALID, "null output handle");
    *out = nullptr;
    if (prec != 32 && prec != 64) return fail(ZC_ERR_INVALID, "precision_bits must be 32 or 64");
    if (n < 1 || n > 48) return fail(ZC_ERR_INVALID, "qubit count must be in 1..=48");
    uint64_t budget = 0;
    int rc = zc_device_budget(0.75, &budget);
    if (rc) return rc;
    return create_state(n, prec, flags, budget, out);
}

namespace zc {
namespace {

// A state's buffers that do not depend on its size: stream, parameter ring
// (pinned host + device), scalar and error words, sampler scratch. Released
// states hand them to a small per-process cache (at most kKitCache, per
// device) and new states take them from it, so a run of short-lived states —
// one zc_run per circuit — does not pay a 32 MiB pinned allocation, a device
// allocation and their frees every time. The cache holds up to
// kKitCache x 64 MiB (half pinned host, half device) until the process exits.
struct Kit {
    int device = 0;
    cudaStream_t stream = nullptr;
    Arena arena;
    double *d_scalar = nullptr, *h_scalar = nullptr;
    int *d_err = nullptr;
    double *d_part = nullptr;
    size_t part_cap = 0;
    void *d_samp = nullptr;
    size_t samp_cap = 0;
};
constexpr size_t kKitCache = 4;
std::mutex g_kit_mu;
std::vector<Kit> g_kits;

void free_kit(Kit &k) {
    if (k.stream) cudaStreamSynchronize(k.stream);
    if (k.arena.host) cudaFreeHost(k.arena.host);
    if (k.arena.dev) cudaFree(k.arena.dev);
    if (k.d_part) cudaFree(k.d_part);
    if (k.d_scalar) cudaFree(k.d_scalar);
    if (k.h_scalar) cudaFreeHost(k.h_scalar);
    if (k.d_samp) cudaFree(k.d_samp);
    if (k.stream) cudaStreamDestroy(k.stream);
    k = Kit{};
}

bool take_kit(int device, Kit *out) {
    std::lock_guard<std::mutex> lk(g_kit_mu);
    for (size_t i = 0; i < g_kits.size(); i++)
        if (g_kits[i].device == device) {
            *out = g_kits[i];
            g_kits.erase(g_kits.begin() + (long)i);
            return true;
        }
    return false;
}

// Returns false when the cache is full (the caller frees the kit).
bool give_kit(const Kit &k) {
    std::lock_guard<std::mutex> lk(g_kit_mu);
    if (g_kits.size() >= kKitCache) return false;
    g_kits.push_back(k);
    return true;
}

}  // namespace
}  // namespace zc

int zc::create_state(uint32_t n, int prec, uint32_t flags, uint64_t budget, zc_state **out) {
    if (!out) return fail(ZC_ERR_INVALID, "null output handle");
    *out = nullptr;
    if (prec != 32 && prec != 64) return fail(ZC_ERR_INVALID, "precision_bits must be 32 or 64");
    if (n < 1 || n > 48) return fail(ZC_ERR_INVALID, "qubit count must be in 1..=48");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(ZC_ERR_UNSUPPORTED, std::string("no usable CUDA device: ") + cudaGetErrorString(e));
    int rc = plan_state(n, prec, budget);
    if (rc) return rc;
    zc_state *st = new zc_state();
    st->n = n;
    st->prec = prec;
    st->flags = flags;
    st->device = dev;
    st->len = 1ull << n;
    st->name = prec == 64 ? "cuda-f64" : "cuda-f32";
    cudaDeviceGetAttribute(&st->num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (st->num_sms <= 0) st->num_sms = 1;
    const size_t bytes = st->len * (prec / 8);
#define TRY(call)                          \
    do {                                   \
        cudaError_t e_ = (call);           \
        if (e_ != cudaSuccess) {           \
            int r_ = cuda_fail(e_, #call); \
            zc_destroy(st);                \
            return r_;                     \
        }                                  \
    } while (0)
    Kit kit;
    if (take_kit(dev, &kit)) {  // stream, ring, scalars, sampler scratch of a released state
        st->stream = kit.stream;
        st->arena = kit.arena;
        st->arena.head = 0;
        st->d_scalar = kit.d_scalar;
        st->h_scalar = kit.h_scalar;
        st->d_err = kit.d_err;
        st->d_part = kit.d_part;
        st->part_cap = kit.part_cap;
        st->d_samp = kit.d_samp;
        st->samp_cap = kit.samp_cap;
    } else {
        TRY(cudaStreamCreateWithFlags(&st->stream, cudaStreamNonBlocking));
    }
    e = cudaMalloc(&st->re, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&st->im, bytes);
    if (e != cudaSuccess) {
        fail(ZC_ERR_MEMORY, std::string("device allocation of the state failed: ") + cudaGetErrorString(e));
        cudaGetLastError();
        zc_destroy(st);
        return ZC_ERR_MEMORY;
    }
    if (!st->arena.host) {
        TRY(cudaMallocHost(&st->arena.host, kArenaBytes));
        TRY(cudaMalloc(&st->arena.dev, kArenaBytes));
        st->arena.cap = kArenaBytes;
        TRY(cudaMalloc(&st->d_scalar, kStatusBytes));
        st->d_err = (int *)((char *)st->d_scalar + kStatusErr);
        TRY(cudaMallocHost(&st->h_scalar, kStatusBytes));
    }
    TRY(cudaMemsetAsync(st->d_scalar, 0, kStatusBytes, st->stream));
#undef TRY
    rc = launch_reset(st);
    if (rc) {
        zc_destroy(st);
        return rc;
    }
    *out = st;
    return ZC_OK;
}

extern "C" {

void zc_destroy(zc_state *st) {
    if (!st) return;
    const bool healthy = !st->stream || cudaStreamSynchronize(st->stream) == cudaSuccess;
    if (st->re) cudaFree(st->re);
    if (st->im) cudaFree(st->im);
    for (auto &r : st->prof_recs) {
        cudaEventDestroy(r.a);
        cudaEventDestroy(r.b);
    }
    for (auto e : st->prof_pool) cudaEventDestroy(e);
    Kit kit;
    kit.device = st->device;
    kit.stream = st->stream;
    kit.arena = st->arena;
    kit.d_scalar = st->d_scalar;
    kit.h_scalar = st->h_scalar;
    kit.d_err = st->d_err;
    kit.d_part = st->d_part;
    kit.part_cap = st->part_cap;
    kit.d_samp = st->d_samp;
    kit.samp_cap = st->samp_cap;
    // a complete kit from a state whose stream finished cleanly goes back to the cache
    const bool complete = kit.stream && kit.arena.host && kit.arena.dev && kit.d_scalar && kit.h_scalar && kit.d_err;
    if (!(healthy && complete && give_kit(kit))) free_kit(kit);
    delete st;
}

const char *zc_name(const zc_state *st) { return st ? st->name.c_str() : ""; }

int zc_apply_unitary(zc_state *st, const uint32_t *qs, uint32_t k, const double *mat) {
    int rc = check_support(st, qs, k, kMaxUnitaryQubits, "apply_unitary");
    if (rc) return rc;
    if (!mat) return fail(ZC_ERR_INVALID, "apply_unitary: null matrix");
    QOp op{Q_UNITARY, k, {}, 0, 0, std::vector<double>(mat, mat + 2 * ((size_t)1 << (2 * k)))};
    for (uint32_t i = 0; i < k; i++) op.qs[i] = qs[i];
    return enqueue(st, std::move(op));
}

int zc_apply_diagonal(zc_state *st, const uint32_t *qs, uint32_t k, const double *d) {
    int rc = check_support(st, qs, k, kMaxDiagQubits, "apply_diagonal");
    if (rc) return rc;
    if (!d) return fail(ZC_ERR_INVALID, "apply_diagonal: null diagonal");
    QOp op{Q_DIAG, k, {}, 0, 0, std::vector<double>(d, d + 2 * ((size_t)1 << k))};
    for (uint32_t i = 0; i < k; i++) op.qs[i] = qs[i];
    return enqueue(st, std::move(op));
}

int zc_apply_cx(zc_state *st, uint32_t c, uint32_t t) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    if (c >= st->n || t >= st->n || c == t) return fail(ZC_ERR_INVALID, "apply_cx: bad control/target");
    return enqueue(st, QOp{Q_CX, 0, {}, c, t, {}});
}

int zc_apply_swap(zc_state *st, uint32_t a, uint32_t b) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    if (a >= st->n || b >= st->n || a == b) return fail(ZC_ERR_INVALID, "apply_swap: bad qubits");
    return enqueue(st, QOp{Q_SWAP, 0, {}, std::min(a, b), std::max(a, b), {}});
}

int zc_prob_one(zc_state *st, uint32_t q, double *out) {
    if (!st || !out) return fail(ZC_ERR_INVALID, "null argument");
    if (q >= st->n) return fail(ZC_ERR_INVALID, "prob_one: qubit out of range");
    int rc = flush(st);
    if (rc) return rc;
    rc = launch_total(st, true, q, exact(st));
    if (rc) return rc;
    return sync_read_scalar(st, out);
}

int zc_measure(zc_state *st, uint32_t q, double u, int *outcome) {
    if (!outcome) return fail(ZC_ERR_INVALID, "null argument");
    double p1 = 0.0;
    int rc = zc_prob_one(st, q, &p1);
    if (rc) return rc;
    const int o = u < p1;
    const double p = o ? p1 : 1.0 - p1;
    rc = launch_collapse(st, q, o, 1.0 / sqrt(p));
    if (rc) return rc;
    *outcome = o;
    return ZC_OK;
}

int zc_reset_all(zc_state *st) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    st->queue.clear();  // queued ops act on a state that is being discarded
    return launch_reset(st);
}

int zc_norm_sqr(zc_state *st, double *out) {
    if (!st || !out) return fail(ZC_ERR_INVALID, "null argument");
    int rc = flush(st);
    if (rc) return rc;
    rc = launch_total(st, false, 0, exact(st));
    if (rc) return rc;
    return sync_read_scalar(st, out);
}

// Backend::sample: pass 1 (chunk masses) and pass 2 (per-chunk rescans) run
// on the GPU, the routing between them on the host.
int zc_sample(zc_state *st, uint64_t shots, uint64_t seed, uint64_t *out) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    if (shots == 0) return ZC_OK;
    if (!out) return fail(ZC_ERR_INVALID, "sample: null output");
    int rc = flush(st);
    if (rc) return rc;
    size_t nch = 0;
    rc = launch_chunk_sums(st, 0, 0, &nch, exact(st));
    if (rc) return rc;
    std::vector<double> sums(nch);
    ZC_CUDA(cudaMemcpyAsync(sums.data(), st->d_part, nch * sizeof(double), cudaMemcpyDeviceToHost, st->stream));
    ZC_CUDA(cudaStreamSynchronize(st->stream));
    SampleRoute route;
    sample_route(sums.data(), nch, st->len, shots, seed, &route);
    rc = grow(&st->d_samp, &st->samp_cap, sample_pass2_bytes(st, route));
    if (rc) return rc;
    uint64_t *d_out = nullptr;
    rc = sample_launch_pass2(st, route, (char *)st->d_samp, &d_out);
    if (rc) return rc;
    ZC_CUDA(cudaMemcpyAsync(out, d_out, shots * sizeof(uint64_t), cudaMemcpyDeviceToHost, st->stream));
    return sync_status(st);
}

int zc_statevector(zc_state *st, double *out) {
    if (!st || !out) return fail(ZC_ERR_INVALID, "null argument");
    int rc = flush(st);
    if (rc) return rc;
    // The device interleaves and widens, a staging buffer at a time, and the
    // copy engine writes the caller's array: 176 GB/s into touched pages. The
    // host touches each piece's pages before its copy, beside the copy of the
    // piece before. Left to the device, the faults of a fresh array took twice
    // as long as that (2^24 amplitudes 17.4 ms, 10.7 here; a host loop over two
    // copied arrays 34) and on one machine thirteen times (223 ms). The staging
    // buffer is the device half of the parameter ring: everything that reads
    // the ring precedes these launches on the stream, everything that refills
    // it follows them.
    const uint64_t chunk = st->arena.cap / (2 * sizeof(double));
    for (uint64_t i = 0; i < st->len; i += chunk) {
        const uint64_t count = std::min<uint64_t>(chunk, st->len - i);
        if ((rc = launch_interleave(st, i, count, st->arena.dev))) return rc;
        touch_pages(out + 2 * i, count * 2 * sizeof(double));
        ZC_CUDA(cudaMemcpyAsync(out + 2 * i, st->arena.dev, count * 2 * sizeof(double), cudaMemcpyDeviceToHost,
                                st->stream));
    }
    return sync_status(st);
}

int zc_load_state(zc_state *st, const double *in) {
    if (!st || !in) return fail(ZC_ERR_INVALID, "null argument");
    st->queue.clear();
    const size_t es = st->prec / 8;
    std::vector<char> re(st->len * es), im(st->len * es);
    for (size_t i = 0; i < st->len; i++) {
        if (st->prec == 64) {
            ((double *)re.data())[i] = in[2 * i];
            ((double *)im.data())[i] = in[2 * i + 1];
        } else {
            ((float *)re.data())[i] = (float)in[2 * i];
            ((float *)im.data())[i] = (float)in[2 * i + 1];
        }
    }
    ZC_CUDA(cudaMemcpyAsync(st->re, re.data(), st->len * es, cudaMemcpyHostToDevice, st->stream));
    ZC_CUDA(cudaMemcpyAsync(st->im, im.data(), st->len * es, cudaMemcpyHostToDevice, st->stream));
    ZC_CUDA(cudaStreamSynchronize(st->stream));
    return ZC_OK;
}

int zc_finish(zc_state *st) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    int rc = flush(st);
    if (rc) return rc;
    ZC_CUDA(cudaGetLastError());
    return sync_status(st);
}

int zc_get_stream(zc_state *st, void **stream) {
    if (!st || !stream) return fail(ZC_ERR_INVALID, "null argument");
    if (hides_queue(st)) {  // what the caller puts on the stream comes behind the ops applied so far
        const int rc = flush(st);
        if (rc) return rc;
        st->stream_out = true;
    }
    *stream = (void *)st->stream;
    return ZC_OK;
}

int zc_profile(zc_state *st, int enable) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    for (auto &r : st->prof_recs) {
        st->prof_pool.push_back(r.a);
        st->prof_pool.push_back(r.b);
    }
    st->prof_recs.clear();
    st->prof = enable != 0;
    return ZC_OK;
}

int zc_profile_read(zc_state *st, zc_kernel_stat *out, int cap, int *n) {
    if (!st || !n) return fail(ZC_ERR_INVALID, "null argument");
    int rc = flush(st);
    if (rc) return rc;
    ZC_CUDA(cudaStreamSynchronize(st->stream));
    zc_kernel_stat agg[K_NKINDS];
    memset(agg, 0, sizeof agg);
    for (const auto &r : st->prof_recs) {
        float ms = 0.f;
        ZC_CUDA(cudaEventElapsedTime(&ms, r.a, r.b));
        agg[r.kind].launches++;
        agg[r.kind].ms += ms;
        agg[r.kind].bytes += r.bytes;
    }
    int m = 0;
    for (int k = 0; k < K_NKINDS; k++) {
        if (!agg[k].launches) continue;
        if (m < cap && out) {
            out[m] = agg[k];
            snprintf(out[m].name, sizeof out[m].name, "%s", kKernelNames[k]);
        }
        m++;
    }
    *n = m;
    return ZC_OK;
}

int zc_set_sweep_shape(zc_state *st, uint32_t max_high) {
    if (!st) return fail(ZC_ERR_INVALID, "null state");
    if (max_high > kMaxSweepHigh) return fail(ZC_ERR_INVALID, "sweep shape: at most 7 high qubits per tile");
    int rc = flush(st);  // queued ops keep the shape they were planned for
    if (rc) return rc;
    st->sweep_high = max_high;
    return ZC_OK;
}

int zc_get_counters(zc_state *st, zc_counters *out) {
    if (!st || !out) return fail(ZC_ERR_INVALID, "null argument");
    if (hides_queue(st)) {
        const int rc = flush(st);
        if (rc) return rc;
    }
    *out = st->ctr;
    return ZC_OK;
}

}  // extern "C"
