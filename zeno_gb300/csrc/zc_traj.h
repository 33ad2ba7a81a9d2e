// Batched trajectory engine: op encoding shared by host and kernel.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace zc {

enum : uint32_t { TOP_GATE = 0, TOP_MEASURE = 1, TOP_RESET = 2 };

// One op of a noisy or dynamic program. Gates: a dense 2^k x 2^k matrix
// (row-major, interleaved re/im f32, at mats + mat_off) on sorted qubits
// qs[0..k); CX and SWAP arrive as permutation matrices, diagonals as dense
// diagonals. mono: every row has exactly one nonzero entry, row r's in column
// (cols >> 3r) & 7. Measure (qubit qs[0] into clbit) and reset (qubit qs[0]) carry
// k = 1 and the identity. `cond` makes the op run only if the classical
// bits [cond_off, cond_off + cond_len) equal cond_value (src/exec.rs:562-566).
struct TrajOp {
    uint32_t k;
    uint32_t qs[3];
    uint32_t mat_off;  // in floats
    uint32_t kind;     // TOP_*
    uint32_t clbit;
    uint32_t cond;
    uint32_t cond_off, cond_len;
    uint64_t cond_value;
    uint32_t mono, cols;
};

// An op with its matrix beside it (k <= 2; three-qubit ops read mats), so
// that a CTA fetches both in one copy of 16-byte pieces.
struct alignas(16) TrajRec {
    TrajOp op;
    float m[32];
};
static_assert(sizeof(TrajRec) % 16 == 0 && sizeof(TrajRec) <= 32 * 16, "one 16-byte piece per lane");

// Launch shape: CTAs, threads per CTA, dynamic shared memory, and the global
// bytes each CTA needs for its state (0: none).
struct TrajPlan {
    int ctas, threads;
    size_t smem;
    size_t global_bytes;
};
constexpr uint64_t kTrajSplitElems = 24576;   // amplitudes held in shared memory at most: 192 KiB of 227
constexpr size_t kTrajSmemMax = 208 * 1024;   // what the kernel may ask for beside its static tables

// NoiseModel fields in src/noise.rs order: dep1q, dep2q, bit flip,
// phase flip, amplitude damping, readout 0->1, readout 1->0.
struct TrajNoise {
    double p[7];
    uint32_t mask;  // bit i: p[i] > 0 (an FP64 comparison takes 64 cycles on the device)
#ifdef __CUDACC__
    __device__ __forceinline__ bool on(int i) const { return (mask >> i) & 1u; }
#endif
};

}  // namespace zc
