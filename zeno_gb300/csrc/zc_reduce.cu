// f64 reductions over the state (norm, prob_one, sampler chunk masses) and
// the sampler's per-chunk resolution pass.
//
// Exact mode keeps the reference's summation order: a serial f64 chain
// inside each 2^16-element chunk (src/sample.rs:38-50, src/state.rs:143-156),
// chunk partials combined serially in chunk order, so norm_sqr, prob_one and
// every sampled index are bit-identical to the CPU oracle for the same state
// bits. The chains are evaluated in parallel with the same roundings
// (zc_chain.h). The sampler's rescan records each chain's value at every
// 32-element stage boundary; draws then resolve in parallel by a binary
// search over those values and a replay of one stage, which repeats the
// chain's own additions bit for bit.
#include <algorithm>

#include "zc_arith.cuh"
#include "zc_chain.h"
#include "zc_internal.h"

namespace zc {
namespace {

// |a|^2 in f64 exactly as `r * r + im * im` after widening (no FMA). On the FP64
// pipe: with the squares on the integer pipe (zc_softmul.h) a 24-qubit circuit
// with every P(1) took 33.1 ms, so 32.6, since a sum waits for its additions.
__device__ __forceinline__ double p2(double r, double i) { return radd(rmul(r, r), rmul(i, i)); }

// Non-negative doubles order like their IEEE bit patterns.
__device__ __forceinline__ unsigned long long dkey(double x) { return (unsigned long long)__double_as_longlong(x); }

constexpr int kChainThreads = 256;
constexpr int kStageElems = 32;  // elements per row: one warp-wide load, one recorded chain value
constexpr int kRowsPerWarp = 8;
constexpr int kTileRows = kRowsPerWarp * kChainThreads / 32;  // 64 rows, two per lane in the scan
constexpr uint64_t kShortChain = 128;  // elements up to which one warp adds a chain up one by one

__device__ __forceinline__ ChainFn shfl_down_fn(const ChainFn &f, int o) {
    return ChainFn{__shfl_down_sync(0xffffffffu, f.a, o), __shfl_down_sync(0xffffffffu, f.b, o)};
}

// One row (32 values, one per lane) as one function of the running mantissa
// in the binade e; capped at kChainCross so that 64 rows add up in 64 bits.
// Lane 0's result counts.
__device__ __forceinline__ ChainFn row_fn(uint64_t vbits, uint32_t e) {
    bool tie;
    const uint64_t k = chain_inc(vbits, e, tie);
    ChainFn f;
    if (__any_sync(0xffffffffu, tie)) {  // ties look at parity: compose in order
        f = chain_fn(k, tie);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) f = chain_then(f, shfl_down_fn(f, o));
    } else {  // plain sum: two 32-bit warp reductions (27 low bits, <= 27 high bits)
        const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)k & 0x7ffffffu);
        const uint32_t hi = __reduce_add_sync(0xffffffffu, (uint32_t)(k >> 27));
        f.a = f.b = ((uint64_t)hi << 27) + lo;
    }
    f.a = f.a < kChainCross ? f.a : kChainCross;
    f.b = f.b < kChainCross ? f.b : kChainCross;
    return f;
}

// One serial f64 chain per CTA (row blockIdx.x), in tiles of 64 rows of 32
// elements. A tile is reduced to one function per row, the rows are scanned
// (every warp repeats the scan: no broadcast barrier), and the first row
// that leaves the accumulator's binade is added serially, after which the
// rows behind it are reduced again in the new binade.
//
// What bounds it: the three FP64 operations per element (|a|^2 must be
// rounded as f64), 60 us per 2^16-element chunk on one SM, with about
// twelve serial rows of 1 us per chunk beside them. One lane per chain, fed
// by producer warps, took 2.9 ms per chunk at any state size (2^16 dependent
// adds of 64 cycles). A chain of up to kShortChain elements crosses a binade in
// nearly every row: one warp adds it up one by one (a draw from an exact 5-qubit
// state 78 -> 57 us; at 256 elements the rows are as fast).
//
// SCAN = false: chunk blockIdx.x of the index space (mode 0: index h; mode 1,
//   prob_one of qubit q: insert_zero(h, q) + 2^q; mode 2: re holds the
//   values themselves); the final chain value goes to part[row].
// SCAN = true: touched chunk cs[row]; the chain starts at the chunk's
//   cum_before and stops once it exceeded the chunk's largest draw;
//   rec[row][stage] holds the chain value at each stage start, rec_nst[row]
//   the stages run and rec_last[row] 1 + the last element with nonzero mass
//   (0: none).
template <typename T, bool SCAN>
__global__ void __launch_bounds__(kChainThreads, 2)
    k_chain(const T *__restrict__ re, const T *__restrict__ im, uint64_t total, uint64_t chunk, int mode, uint32_t q,
            const SampleChunk *__restrict__ cs, const double *__restrict__ us, double *__restrict__ part,
            double *__restrict__ rec, uint32_t *__restrict__ rec_nst, unsigned long long *__restrict__ rec_last,
            uint32_t rec_stride) {
    __shared__ ChainFn s_row[2][kTileRows];  // double-buffered: one barrier per scan
    __shared__ uint64_t s_acc;
    __shared__ unsigned long long s_last;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint64_t row = blockIdx.x;
    uint64_t c = row, acc = 0;
    unsigned long long stop = ~0ull, my_last = 0;
    if (SCAN) {
        const SampleChunk sc = cs[row];
        c = sc.chunk;
        acc = dkey(sc.cum);
        stop = dkey(us[sc.s1 - 1]);
        if (threadIdx.x == 0) s_last = 0;
    }
    const uint64_t first = c * chunk, len = total - first < chunk ? total - first : chunk;
    const uint64_t sbit = 1ull << q;
    const uint32_t nst = (uint32_t)((len + kStageElems - 1) / kStageElems);
    if (len <= kShortChain) {
        if (warp) return;
        double a = __longlong_as_double((long long)acc);
        auto value = [&](uint32_t r) {
            const uint64_t e = (uint64_t)r * kStageElems + lane, h = first + e;
            if (e >= len) return 0ull;
            const uint64_t idx = mode == 1 ? insert_zero(h, q) + sbit : h;
            return dkey(mode == 2 ? widen(re[idx]) : p2(widen(re[idx]), widen(im[idx])));
        };
        unsigned long long v = value(0);
        for (uint32_t r = 0; r < nst; r++) {
            const unsigned long long next = r + 1 < nst ? value(r + 1) : 0ull;
            if (SCAN) {
                if (lane == 0) rec[row * rec_stride + r] = a;
                const uint32_t mass = __ballot_sync(0xffffffffu, v != 0ull);
                if (mass) my_last = (unsigned long long)r * kStageElems + 32 - __clz(mass);
            }
#pragma unroll 8
            for (int i = 0; i < 32; i++)
                a = radd(a, __longlong_as_double((long long)__shfl_sync(0xffffffffu, v, i)));
            v = next;
        }
        if (lane == 0) {
            if (SCAN) {
                rec_nst[row] = nst;
                rec_last[row] = my_last;
            } else {
                part[row] = a;
            }
        }
        return;
    }
    uint32_t ran = nst;
    T nr[kRowsPerWarp], ni[kRowsPerWarp];  // the next tile's amplitudes, in flight while this one is summed
    auto fetch = [&](uint64_t t0) {
#pragma unroll
        for (int j = 0; j < kRowsPerWarp; j++) {
            const uint64_t e = t0 + (uint64_t)((warp * kRowsPerWarp + j) * kStageElems + lane);
            nr[j] = ni[j] = (T)0;
            if (e < len) {
                const uint64_t h = first + e;
                const uint64_t idx = mode == 1 ? insert_zero(h, q) + sbit : h;
                nr[j] = re[idx];
                if (mode != 2) ni[j] = im[idx];
            }
        }
    };
    int buf = 0;
    fetch(0);
    for (uint64_t t0 = 0; t0 < len; t0 += kTileRows * kStageElems) {
        uint64_t v[kRowsPerWarp];
#pragma unroll
        for (int j = 0; j < kRowsPerWarp; j++) {
            v[j] = dkey(mode == 2 ? widen(nr[j]) : p2(widen(nr[j]), widen(ni[j])));
            if (SCAN && v[j]) my_last = t0 + (uint64_t)((warp * kRowsPerWarp + j) * kStageElems + lane) + 1;
        }
        if (t0 + kTileRows * kStageElems < len) fetch(t0 + kTileRows * kStageElems);
        for (int from = 0; from < kTileRows;) {
            uint32_t e;
            uint64_t m;
            chain_split(acc, e, m);
            buf ^= 1;
#pragma unroll
            for (int j = 0; j < kRowsPerWarp; j++) {
                const int r = warp * kRowsPerWarp + j;
                ChainFn f{0, 0};
                if (r >= from) f = row_fn(v[j], e);
                if (lane == 0) s_row[buf][r] = f;
            }
            __syncthreads();
            const ChainFn f0 = s_row[buf][2 * lane], f1 = s_row[buf][2 * lane + 1];
            ChainFn g = chain_then(f0, f1);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const ChainFn h{__shfl_up_sync(0xffffffffu, g.a, o), __shfl_up_sync(0xffffffffu, g.b, o)};
                if (lane >= o) g = chain_then(h, g);
            }
            ChainFn ex{__shfl_up_sync(0xffffffffu, g.a, 1), __shfl_up_sync(0xffffffffu, g.b, 1)};
            if (lane == 0) ex = ChainFn{0, 0};
            const uint64_t m0 = chain_apply(ex, m), m1 = chain_apply(f0, m0), m2 = chain_apply(f1, m1);
            const uint32_t c1 = __ballot_sync(0xffffffffu, m1 >= kChainCross);
            const uint32_t c2 = __ballot_sync(0xffffffffu, m2 >= kChainCross);
            int x = kTileRows;  // the first row that leaves the binade
            if (c1 | c2) {
                const int l = __ffs(c1 | c2) - 1;
                x = 2 * l + (int)(((c1 >> l) & 1u) ^ 1u);
            }
            if (SCAN && warp == 0) {
                const uint32_t st0 = (uint32_t)(t0 / kStageElems);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = 2 * lane + h;
                    if (r >= from && r <= x && st0 + r < nst)
                        rec[row * rec_stride + st0 + r] = __longlong_as_double((long long)chain_pack(e, h ? m1 : m0));
                }
            }
            if (x == kTileRows) {
                acc = chain_pack(e, __shfl_sync(0xffffffffu, m2, 31));
                break;
            }
            const uint64_t ax = __shfl_sync(0xffffffffu, (x & 1) ? m1 : m0, x >> 1);
            if (warp == x / kRowsPerWarp) {
                uint64_t vx = 0;
#pragma unroll
                for (int j = 0; j < kRowsPerWarp; j++)
                    vx |= x % kRowsPerWarp == j ? v[j] : 0;
                double a = __longlong_as_double((long long)chain_pack(e, ax));
#pragma unroll 8
                for (int i = 0; i < 32; i++)
                    a = radd(a, __longlong_as_double((long long)__shfl_sync(0xffffffffu, vx, i)));
                if (lane == 0) s_acc = dkey(a);
            }
            __syncthreads();
            acc = s_acc;
            from = x + 1;
        }
        if (SCAN && acc > stop) {
            const uint64_t done = (t0 / kStageElems) + kTileRows;
            ran = done < nst ? (uint32_t)done : nst;
            break;
        }
    }
    if (SCAN) {
        if (my_last) atomicMax(&s_last, my_last);
        __syncthreads();
        if (threadIdx.x == 0) {
            rec_nst[row] = ran;
            rec_last[row] = s_last;
        }
    } else if (threadIdx.x == 0) {
        part[row] = __longlong_as_double((long long)acc);
    }
}

// Sampler pass 2 resolution (src/sample.rs:64-108), blockIdx.x a touched
// chunk, one thread per draw: the draw lands in the last stage t whose start
// value is <= u; replaying stage t's additions from that value gives the
// first index i with u < acc_i, the index the serial rescan emits. A draw
// never exceeded by the chain goes to the chunk's last index with nonzero
// mass (its last index if none).
// A replay costs up to 128 FP64 operations, so the draws of a chunk are
// spread over blockIdx.y when there are few chunks: 1000 draws of one chunk
// keep one SM's FP64 pipe busy for 40 us, 32 SMs' for 1.
constexpr int kResolveThreads = 32;

template <typename T>
__global__ void __launch_bounds__(kResolveThreads) k_resolve(const T *__restrict__ re, const T *__restrict__ im,
                                                 const SampleChunk *__restrict__ cs, const double *__restrict__ us,
                                                 uint64_t *__restrict__ out, uint64_t chunk_len, uint64_t total,
                                                 const double *__restrict__ rec, const uint32_t *__restrict__ rec_nst,
                                                 const unsigned long long *__restrict__ rec_last,
                                                 uint32_t rec_stride) {
    const uint64_t b = blockIdx.x;
    const SampleChunk sc = cs[b];
    const uint64_t first = sc.chunk * chunk_len;
    const uint64_t len = total - first < chunk_len ? total - first : chunk_len;
    const uint32_t n = rec_nst[b];
    const double *A = rec + b * rec_stride;
    for (uint64_t d = sc.s0 + blockIdx.y * blockDim.x + threadIdx.x; d < sc.s1; d += gridDim.y * blockDim.x) {
        const unsigned long long uk = dkey(us[d]);
        uint32_t lo = 0, hi = n - 1;  // A[0] = cum_before <= u by the host's routing
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) / 2;
            if (dkey(A[mid]) <= uk) lo = mid;
            else hi = mid - 1;
        }
        double acc = A[lo];
        const uint64_t e0 = (uint64_t)lo * kStageElems;
        const uint64_t e1 = e0 + kStageElems < len ? e0 + kStageElems : len;
        uint64_t res = ~0ull;
        for (uint64_t e = e0; e < e1 && res == ~0ull; e += 4) {  // four loads in flight
            double v[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                v[j] = e + j < e1 ? p2(widen(re[first + e + j]), widen(im[first + e + j])) : 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc = radd(acc, v[j]);
                if (res == ~0ull && uk < dkey(acc)) res = first + e + j;
            }
        }
        if (res == ~0ull) res = rec_last[b] ? first + rec_last[b] - 1 : first + len - 1;
        out[d] = res;
    }
}

// ------------------------------------------------------------------
// Fast mode (ZC_FLAG_FAST): the same quantities as parallel double-float
// reductions on the FP32 pipe (~2^-46 relative error per step instead of
// the reference's serial f64 order). Chunk boundaries and the host routing
// of draws are the exact path's; only the order of additions inside a
// chunk differs, so a draw can move by one index only where it falls
// within rounding distance of a cumulative boundary.

// a + b in double-float (TwoSum on the high parts, low parts summed).
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
    float e;
    const float s = two_sum(a.x, b.x, e);
    return df_norm(s, __fadd_rn(e, __fadd_rn(a.y, b.y)));
}

__device__ __forceinline__ float2 p2_df(double r, double i) {
    const float2 a = df_from_f64(r), b = df_from_f64(i);
    return df_dot2(a, a, b, b);
}

__device__ __forceinline__ float2 p2_df(float r, float i) {
    const float2 a = make_float2(r, 0.f), b = make_float2(i, 0.f);
    return df_dot2(a, a, b, b);
}

__device__ __forceinline__ float2 shfl_xor_df(float2 v, int m) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

__device__ __forceinline__ float2 shfl_up_df(float2 v, int d) {
    return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}

// Non-negative value as an order-preserving integer key (IEEE bits of f64).
__device__ __forceinline__ unsigned long long df_key(float2 v) {
    return (unsigned long long)__double_as_longlong(df_to_f64(v));
}

constexpr int kDfThreads = 256;

// CTA-wide double-float sum; every thread gets the result. `red` holds 8 slots.
__device__ __forceinline__ float2 block_sum_df(float2 v, float2 *red) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v = df_add(v, shfl_xor_df(v, m));
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float2 t = make_float2(0.f, 0.f);
    for (int w = 0; w < (int)(blockDim.x / 32); w++) t = df_add(t, red[w]);
    return t;
}

// One CTA per chunk; f64 partials (the sampler's chunk masses).
// NT threads: 1024 while the chunks leave SMs idle, where a chunk's latency is
// what counts (wide_chunks), else 256.
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_chunk_sums_df(const T *__restrict__ re, const T *__restrict__ im,
                                                      uint64_t total, uint64_t chunk, double *__restrict__ part) {
    __shared__ float2 red[NT / 32];
    const uint64_t lo = (uint64_t)blockIdx.x * chunk;
    const uint64_t hi = lo + chunk < total ? lo + chunk : total;
    float2 acc[4] = {};
    for (uint64_t h0 = lo + threadIdx.x; h0 < hi; h0 += 4 * NT) {
        T vr[4], vi[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t h = h0 + (uint64_t)u * NT;
            vr[u] = vi[u] = (T)0;
            if (h < hi) {
                vr[u] = re[h];
                vi[u] = im[h];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) acc[u] = df_add(acc[u], p2_df(vr[u], vi[u]));
    }
    const float2 t = block_sum_df(df_add(df_add(acc[0], acc[1]), df_add(acc[2], acc[3])), red);
    if (threadIdx.x == 0) part[blockIdx.x] = df_to_f64(t);
}

// The whole sum (norm_sqr; ONES: the q = 1 half, prob_one) in one launch: CTAs
// stride over 16-byte vectors, four in flight per thread and array, and the
// last one to finish (a ticket) adds the CTAs' partials. A qubit whose halves
// alternate inside a vector reads everything and keeps its elements; DRAM
// moves whole sectors either way.
// Bound by HBM. One CTA per 2^16 elements and a second launch took 124 us for
// prob_one at 25 qubits (f64, 268 MB), this and one readback instead of two 79.
template <typename T, bool ONES>
__global__ void __launch_bounds__(kDfThreads) k_total_df(const T *__restrict__ re, const T *__restrict__ im,
                                                         uint64_t units, uint32_t q, double *__restrict__ part,
                                                         unsigned *__restrict__ ticket, double *__restrict__ out) {
    __shared__ float2 red[kDfThreads / 32];
    __shared__ bool s_last;
    using VT = typename Vec<T>::type;
    constexpr int V = Vec<T>::N, U = 4;
    const bool inside = ONES && (1ull << q) < (uint64_t)V;  // both halves in every vector
    const uint64_t stride = (uint64_t)gridDim.x * kDfThreads;
    float2 acc[U] = {};
    auto element = [&](uint64_t u) {  // first element of vector u of the sum
        return ONES && !inside ? insert_zero(u * V, q) + (1ull << q) : u * V;
    };
    for (uint64_t u0 = blockIdx.x * (uint64_t)kDfThreads + threadIdx.x; u0 < units; u0 += U * stride) {
        VT vr[U], vi[U];
#pragma unroll
        for (int k = 0; k < U; k++)
            if (u0 + k * stride < units) {
                const uint64_t i = element(u0 + k * stride);
                vr[k] = *reinterpret_cast<const VT *>(re + i);
                vi[k] = *reinterpret_cast<const VT *>(im + i);
            }
#pragma unroll
        for (int k = 0; k < U; k++)
            if (u0 + k * stride < units) {
                const T *r = reinterpret_cast<const T *>(&vr[k]), *m = reinterpret_cast<const T *>(&vi[k]);
#pragma unroll
                for (int e = 0; e < V; e++)
                    if (!inside || ((e >> q) & 1)) acc[k] = df_add(acc[k], p2_df(r[e], m[e]));
            }
    }
    const float2 t = block_sum_df(df_add(df_add(acc[0], acc[1]), df_add(acc[2], acc[3])), red);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = df_to_f64(t);
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float2 a = make_float2(0.f, 0.f);
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += kDfThreads) a = df_add(a, df_from_f64(__ldcg(part + i)));
    const float2 sum = block_sum_df(a, red);
    if (threadIdx.x == 0) {
        *out = df_to_f64(sum);
        *ticket = 0;  // for the next launch on this stream
    }
}

template <typename T>
__global__ void k_total_small(const T *re, const T *im, uint64_t total, int ones, uint32_t q, double *out) {
    float2 a = make_float2(0.f, 0.f);  // states shorter than a vector
    for (uint64_t h = 0; h < total; h++) {
        const uint64_t i = ones ? insert_zero(h, q) + (1ull << q) : h;
        a = df_add(a, p2_df(re[i], im[i]));
    }
    *out = df_to_f64(a);
}

// Sampler pass 2, one CTA per touched chunk: tiles of NT x 8 or 4
// elements get a
// CTA-wide inclusive prefix of |a|^2 (double-float) on top of the running
// cumulative; each draw of the tile resolves by binary search to the first
// index whose cumulative exceeds it (the reference's `us[ptr] < acc`).
// Draws left over past the chunk go to its last nonzero index.
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_sample_scan_df(const T *__restrict__ re, const T *__restrict__ im,
                                                               const SampleChunk *__restrict__ cs,
                                                               const double *__restrict__ us,
                                                               uint64_t *__restrict__ out, uint64_t chunk_len,
                                                               uint64_t total) {
    constexpr int kScanPer = NT == 1024 ? 4 : 8, kScanTile = NT * kScanPer;
    __shared__ float2 s_cum[kScanTile];
    __shared__ float2 s_wsum[NT / 32];
    __shared__ unsigned long long s_last;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const SampleChunk sc = cs[blockIdx.x];
    const uint64_t lo = sc.chunk * chunk_len;
    const uint64_t hi = lo + chunk_len < total ? lo + chunk_len : total;
    uint64_t ptr = sc.s0;
    float2 base = df_from_f64<true>(sc.cum);  // never above the host's cum
    unsigned long long my_last = 0;     // 1 + last index with nonzero mass seen
    for (uint64_t t0 = lo; t0 < hi && ptr < sc.s1; t0 += kScanTile) {
        const uint64_t e0 = t0 + (uint64_t)tid * kScanPer;
        float2 pre[kScanPer];
        float2 run = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < kScanPer; j++) {
            const uint64_t i = e0 + j;
            float2 p = make_float2(0.f, 0.f);
            if (i < hi) {
                p = p2_df(re[i], im[i]);
                if (p.x > 0.f) my_last = i + 1;
            }
            run = df_add(run, p);
            pre[j] = run;
        }
        float2 incl = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float2 v = shfl_up_df(incl, d);
            if (lane >= d) incl = df_add(v, incl);
        }
        float2 excl = shfl_up_df(incl, 1);
        if (lane == 0) excl = make_float2(0.f, 0.f);
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        float2 wpre = make_float2(0.f, 0.f);
        if constexpr (NT == 1024) {  // 32 warps: a scan, not 31 sums in a row
            float2 ws = s_wsum[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const float2 v = shfl_up_df(ws, d);
                if (lane >= d) ws = df_add(v, ws);
            }
            const int from = warp ? warp - 1 : 0;
            const float2 before = make_float2(__shfl_sync(0xffffffffu, ws.x, from), __shfl_sync(0xffffffffu, ws.y, from));
            if (warp) wpre = before;
        } else {
            for (int w = 0; w < warp; w++) wpre = df_add(wpre, s_wsum[w]);
        }
        const float2 tb = df_add(base, df_add(wpre, excl));
#pragma unroll
        for (int j = 0; j < kScanPer; j++) s_cum[tid * kScanPer + j] = df_add(tb, pre[j]);
        __syncthreads();
        const int nvalid = hi - t0 < (uint64_t)kScanTile ? (int)(hi - t0) : kScanTile;
        const unsigned long long end_key = df_key(s_cum[nvalid - 1]);
        uint64_t resolved = 0;
        for (uint64_t d0 = ptr; d0 < sc.s1; d0 += NT) {
            const uint64_t d = d0 + tid;
            int in = 0;
            if (d < sc.s1) {
                const unsigned long long uk = (unsigned long long)__double_as_longlong(us[d]);
                if (uk < end_key) {
                    in = 1;
                    int a = 0, b = nvalid - 1;  // first j with key(cum_j) > u; j = nvalid-1 qualifies
                    while (a < b) {
                        const int m = (a + b) / 2;
                        if (df_key(s_cum[m]) > uk) b = m;
                        else a = m + 1;
                    }
                    out[d] = t0 + (uint64_t)a;
                }
            }
            const int cnt = __syncthreads_count(in);
            resolved += (uint64_t)cnt;
            if (cnt < NT) break;
        }
        ptr += resolved;
        base = s_cum[nvalid - 1];
        __syncthreads();  // s_cum and s_wsum are rewritten by the next tile
    }
    if (ptr < sc.s1) {
        if (tid == 0) s_last = 0;
        __syncthreads();
        if (my_last) atomicMax(&s_last, my_last);
        __syncthreads();
        const uint64_t ln = s_last ? s_last - 1 : hi - 1;
        for (uint64_t d = ptr + tid; d < sc.s1; d += NT) out[d] = ln;
    }
}

// Launch k_chain, one CTA per chain; rec != nullptr selects SCAN.
template <typename T, bool SCAN>
int run_chain(zc_state *st, uint64_t total, uint64_t chunk, uint64_t nrows, int mode, uint32_t q,
              const SampleChunk *cs, const double *us, double *part, double *rec, uint32_t stride) {
    unsigned long long *rec_last = nullptr;
    uint32_t *rec_nst = nullptr;
    if (SCAN) {
        rec_last = (unsigned long long *)(rec + nrows * stride);
        rec_nst = (uint32_t *)(rec_last + nrows);
    }
    k_chain<T, SCAN><<<(unsigned)nrows, kChainThreads, 0, st->stream>>>((const T *)st->re, (const T *)st->im, total,
                                                                       chunk, mode, q, cs, us, part, rec, rec_nst,
                                                                       rec_last, stride);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

// Split re / im arrays -> interleaved f64 (re, im) pairs, four amplitudes per
// thread (16-byte loads, 64 bytes of stores).
template <typename T>
__global__ void __launch_bounds__(256) k_interleave(const T *__restrict__ re, const T *__restrict__ im,
                                                    double2 *__restrict__ out, uint64_t len) {
    const uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 4;
    if (i + 4 <= len) {
        using VT = typename Vec<T>::type;
        constexpr int V = Vec<T>::N;
        VT vr[4 / V], vm[4 / V];
#pragma unroll
        for (int k = 0; k < 4 / V; k++) {
            vr[k] = reinterpret_cast<const VT *>(re + i)[k];
            vm[k] = reinterpret_cast<const VT *>(im + i)[k];
        }
        const T *r = reinterpret_cast<const T *>(vr), *m = reinterpret_cast<const T *>(vm);
#pragma unroll
        for (int k = 0; k < 4; k++) out[i + k] = make_double2(widen(r[k]), widen(m[k]));
    } else {
        for (uint64_t k = i; k < len; k++) out[k] = make_double2(widen(re[k]), widen(im[k]));
    }
}

}  // namespace

int launch_interleave(zc_state *st, uint64_t first, uint64_t count, void *dst) {
    const unsigned blocks = (unsigned)((count + 1023) / 1024);
    st->ctr.launches++;
    if (st->prec == 64)
        k_interleave<double><<<blocks, 256, 0, st->stream>>>((const double *)st->re + first,
                                                             (const double *)st->im + first, (double2 *)dst, count);
    else
        k_interleave<float><<<blocks, 256, 0, st->stream>>>((const float *)st->re + first,
                                                            (const float *)st->im + first, (double2 *)dst, count);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

// Chunks enough for two CTAs of 256 threads per SM keep HBM busy (30q: 93-97%
// of its peak); fewer are as fast as one chunk, which 1024 threads take through
// sooner: 1024 draws at 19 qubits (8 chunks) within a run of 1.63 -> 1.48 ms,
// 24 served requests 7.4 -> 6.9 ms; 25 qubits (512 chunks) unchanged.
// (States of up to 4096 amplitudes are a few vectors per thread: 256 threads, 8
// qubits 64 -> 57 us.)
static bool wide_chunks(const zc_state *st, size_t nch) {
    return nch <= (size_t)st->num_sms * 2 && st->len > 4096;
}

template <typename T>
void run_chunk_sums_df(zc_state *st, uint64_t total, uint64_t chunk, size_t nch, double *part) {
    const T *re = (const T *)st->re, *im = (const T *)st->im;
    if (wide_chunks(st, nch)) k_chunk_sums_df<T, 1024><<<(unsigned)nch, 1024, 0, st->stream>>>(re, im, total, chunk, part);
    else k_chunk_sums_df<T, kDfThreads><<<(unsigned)nch, kDfThreads, 0, st->stream>>>(re, im, total, chunk, part);
}

template <typename T>
void run_sample_scan_df(zc_state *st, size_t nch, const SampleChunk *cs, const double *us, uint64_t *out,
                        uint64_t chunk_len) {
    const T *re = (const T *)st->re, *im = (const T *)st->im;
    if (wide_chunks(st, nch))
        k_sample_scan_df<T, 1024><<<(unsigned)nch, 1024, 0, st->stream>>>(re, im, cs, us, out, chunk_len, st->len);
    else
        k_sample_scan_df<T, kDfThreads><<<(unsigned)nch, kDfThreads, 0, st->stream>>>(re, im, cs, us, out, chunk_len, st->len);
}

// The partial sums' buffer, at least `count` long. Its capacity is zero while
// there is none: one left over from before a failed allocation would send the
// next, smaller sum to a null pointer.
static int grow_part(zc_state *st, size_t count) {
    if (count <= st->part_cap) return ZC_OK;
    if (st->d_part) cudaFree(st->d_part);
    st->d_part = nullptr;
    st->part_cap = 0;
    ZC_CUDA(cudaMalloc(&st->d_part, count * sizeof(double)));
    st->part_cap = count;
    return ZC_OK;
}

int launch_chunk_sums(zc_state *st, int mode, uint32_t q, size_t *nchunks_out, bool exact, double *out) {
    const uint64_t total = mode == 0 ? st->len : st->len / 2;
    const uint64_t chunk = total < (1ull << kSampleChunkLog2) ? total : (1ull << kSampleChunkLog2);
    const uint64_t nch = (total + chunk - 1) / chunk;
    if (!out) {
        const int rc = grow_part(st, nch);
        if (rc) return rc;
    }
    double *part = out ? out : st->d_part;
    ProfScope ps(st, K_CHUNK_SUMS, (mode == 0 ? 1.0 : 0.5) * st->len * (st->prec / 8) * 2);
    st->ctr.launches++;
    *nchunks_out = nch;
    if (!exact) {  // only whole-state masses: prob_one is launch_total's
        if (mode != 0) return fail(ZC_ERR_INVALID, "fast chunk sums cover whole states");
        if (st->prec == 64) run_chunk_sums_df<double>(st, total, chunk, nch, part);
        else run_chunk_sums_df<float>(st, total, chunk, nch, part);
        ZC_CUDA(cudaGetLastError());
        return ZC_OK;
    }
    if (st->prec == 64)
        return run_chain<double, false>(st, total, chunk, nch, mode, q, nullptr, nullptr, part, nullptr, 0);
    return run_chain<float, false>(st, total, chunk, nch, mode, q, nullptr, nullptr, part, nullptr, 0);
}

template <typename T>
int run_total(zc_state *st, bool ones, uint32_t q) {
    constexpr uint64_t V = Vec<T>::N;
    const T *re = (const T *)st->re, *im = (const T *)st->im;
    unsigned *ticket = (unsigned *)((char *)st->d_scalar + kStatusTicket);
    if (st->len < 2 * V) {
        k_total_small<T><<<1, 1, 0, st->stream>>>(re, im, ones ? st->len / 2 : st->len, ones, q, st->d_scalar);
    } else {
        const uint64_t units = (ones && (1ull << q) >= V ? st->len / 2 : st->len) / V;
        const uint64_t want = (units + kDfThreads - 1) / kDfThreads, cap = (uint64_t)st->num_sms * 8;
        const unsigned blocks = (unsigned)std::min(want, cap);
        const int rc = blocks > st->part_cap ? grow_part(st, cap) : ZC_OK;
        if (rc) return rc;
        if (ones) k_total_df<T, true><<<blocks, kDfThreads, 0, st->stream>>>(re, im, units, q, st->d_part, ticket, st->d_scalar);
        else k_total_df<T, false><<<blocks, kDfThreads, 0, st->stream>>>(re, im, units, q, st->d_part, ticket, st->d_scalar);
    }
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

int launch_total(zc_state *st, bool ones, uint32_t q, bool exact) {
    if (exact) {  // chunk chains, then the chunks in order
        size_t nch = 0;
        const int rc = launch_chunk_sums(st, ones ? 1 : 0, q, &nch, true);
        if (rc) return rc;
        ProfScope ps(st, K_SERIAL_SUM, 8.0 * nch);
        st->ctr.launches++;
        k_chain<double, false><<<1, kChainThreads, 0, st->stream>>>(st->d_part, nullptr, nch, nch, 2, 0, nullptr,
                                                                    nullptr, st->d_scalar, nullptr, nullptr, nullptr,
                                                                    0);
        ZC_CUDA(cudaGetLastError());
        return ZC_OK;
    }
    ProfScope ps(st, K_CHUNK_SUMS, (ones ? 0.5 : 1.0) * st->len * (st->prec / 8) * 2);
    st->ctr.launches++;
    return st->prec == 64 ? run_total<double>(st, ones, q) : run_total<float>(st, ones, q);
}

int launch_sample_scan(zc_state *st, const SampleChunk *d_chunks, size_t nchunks, const double *d_us,
                       uint64_t *d_out, uint64_t chunk_len, bool exact, void *d_scratch) {
    if (nchunks == 0) return ZC_OK;
    ProfScope ps(st, K_SAMPLE_SCAN, (double)nchunks * chunk_len * (st->prec / 8) * 2);
    st->ctr.launches++;
    if (!exact) {
        if (st->prec == 64) run_sample_scan_df<double>(st, nchunks, d_chunks, d_us, d_out, chunk_len);
        else run_sample_scan_df<float>(st, nchunks, d_chunks, d_us, d_out, chunk_len);
        ZC_CUDA(cudaGetLastError());
        return ZC_OK;
    }
    const uint32_t stride = (uint32_t)((chunk_len + kStageElems - 1) / kStageElems);
    double *rec = (double *)d_scratch;
    unsigned long long *rec_last = (unsigned long long *)(rec + nchunks * stride);
    uint32_t *rec_nst = (uint32_t *)(rec_last + nchunks);
    int rc = st->prec == 64 ? run_chain<double, true>(st, st->len, chunk_len, nchunks, 0, 0, d_chunks, d_us, nullptr,
                                                      rec, stride)
                            : run_chain<float, true>(st, st->len, chunk_len, nchunks, 0, 0, d_chunks, d_us, nullptr,
                                                     rec, stride);
    if (rc) return rc;
    // about eight CTAs per SM in all; those past a chunk's draws exit at once
    const uint64_t split = std::max<uint64_t>(1, (uint64_t)st->num_sms * 8 / nchunks);
    const dim3 grid((unsigned)nchunks, (unsigned)std::min<uint64_t>(split, 256));
    if (st->prec == 64)
        k_resolve<double><<<grid, kResolveThreads, 0, st->stream>>>((const double *)st->re, (const double *)st->im,
                                                                    d_chunks, d_us, d_out, chunk_len, st->len, rec,
                                                                    rec_nst, rec_last, stride);
    else
        k_resolve<float><<<grid, kResolveThreads, 0, st->stream>>>((const float *)st->re, (const float *)st->im,
                                                                   d_chunks, d_us, d_out, chunk_len, st->len, rec,
                                                                   rec_nst, rec_last, stride);
    ZC_CUDA(cudaGetLastError());
    return ZC_OK;
}

size_t sample_scan_scratch(size_t nchunks, uint64_t chunk_len, bool exact) {
    if (!exact) return 0;
    const size_t stride = (chunk_len + kStageElems - 1) / kStageElems;
    return nchunks * (stride * sizeof(double) + sizeof(unsigned long long) + sizeof(uint32_t)) + 256;
}

}  // namespace zc
