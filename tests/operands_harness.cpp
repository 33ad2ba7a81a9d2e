// Host check that a sweep job whose operands leave the tile, the state or the
// tables is refused when it is encoded (zeno_gb300/csrc/zc_sweep.cu
// encode_job): the kernel indexes with them unchecked. Links the built
// libzeno_cuda.so; no GPU.
#include <cstdio>
#include <functional>
#include <vector>

#include "zc_internal.h"

using zc::MicroOp;

// A tile of 2^8 slots of a 12-qubit state (five row bits, three high qubits).
static zc::SweepPlan plan_of(const MicroOp &m, size_t table_bytes) {
    zc::SweepPlan p;
    p.g = zc::SweepGeom{};
    p.g.n = 12;
    p.g.L = 5;
    p.g.H = 3;
    for (uint32_t j = 0; j < 3; j++) p.g.hpos[j] = 7 + j;
    p.g.ntiles = 16;
    p.mops = {m};
    p.tables.assign(table_bytes, 0);
    return p;
}

int main() {
    const uint32_t O = zc::kOuterFlag;
    MicroOp base{};
    int n_ok = 0, n_bad = 0;
    for (int prec : {32, 64})
        for (bool exact : {false, true}) {
            const bool df = prec == 64 && !exact;
            const size_t entry = prec == 64 ? 16 : 8;
            auto expect = [&](bool good, const char *what, uint32_t kind, std::function<void(MicroOp &)> set,
                              size_t table = 0) {
                MicroOp m = base;
                m.kind = kind;
                set(m);
                std::vector<char> out;
                const bool ok = zc::encode_job(prec, exact, plan_of(m, table), &out) == ZC_OK;
                if (ok != good) std::printf("FAIL %s (f%d, %s)\n", what, prec, exact ? "exact" : "fast");
                (good ? n_ok : n_bad)++;
                return ok == good;
            };
            auto ab = [](uint32_t a, uint32_t b) {
                return [=](MicroOp &m) {
                    m.a = a;
                    m.b = b;
                };
            };
            auto dk = [](std::vector<uint32_t> loc, uint64_t table) {
                return [=](MicroOp &m) {
                    m.k = (uint32_t)loc.size();
                    for (size_t i = 0; i < loc.size() && i < 12; i++) m.loc[i] = loc[i];
                    m.table = table;
                };
            };
            bool ok = true;
            for (uint32_t kind : std::vector<uint32_t>{zc::MOP_U1, zc::MOP_R1, zc::MOP_RT}) {
                if (kind != zc::MOP_U1 && !df) continue;
                ok &= expect(true, "gate", kind, ab(7, 0));
                ok &= expect(false, "gate bit above the tile", kind, ab(8, 0));
                ok &= expect(false, "gate on an outer qubit", kind, ab(O | 5, 0));
            }
            if (!df) {
                ok &= expect(true, "diagonal", zc::MOP_D1, ab(7, 0));
                ok &= expect(true, "outer diagonal", zc::MOP_D1, ab(O | 11, 0));
                ok &= expect(false, "diagonal above the tile", zc::MOP_D1, ab(8, 0));
                ok &= expect(false, "diagonal beyond the state", zc::MOP_D1, ab(O | 12, 0));
            }
            ok &= expect(true, "CX", zc::MOP_CX, ab(0, 7));
            ok &= expect(true, "outer control", zc::MOP_CX, ab(O | 11, 7));
            ok &= expect(false, "control above the tile", zc::MOP_CX, ab(8, 0));
            ok &= expect(false, "control beyond the state", zc::MOP_CX, ab(O | 12, 0));
            ok &= expect(false, "target above the tile", zc::MOP_CX, ab(0, 8));
            ok &= expect(false, "outer target", zc::MOP_CX, ab(0, O | 5));
            ok &= expect(false, "control on the target", zc::MOP_CX, ab(3, 3));
            ok &= expect(true, "SWAP", zc::MOP_SWAP, ab(0, 7));
            ok &= expect(false, "SWAP above the tile", zc::MOP_SWAP, ab(8, 0));
            ok &= expect(false, "SWAP above the tile, second", zc::MOP_SWAP, ab(0, 8));
            ok &= expect(false, "SWAP with an outer qubit", zc::MOP_SWAP, ab(O | 5, 0));
            ok &= expect(false, "SWAP with itself", zc::MOP_SWAP, ab(2, 2));
            ok &= expect(true, "table", zc::MOP_DK, dk({0, 7, O | 11}, 16), 16 + 8 * entry);
            ok &= expect(false, "table location above the tile", zc::MOP_DK, dk({0, 8, O | 11}, 16), 16 + 8 * entry);
            ok &= expect(false, "table location beyond the state", zc::MOP_DK, dk({0, 7, O | 12}, 16), 16 + 8 * entry);
            ok &= expect(false, "table beyond the tables", zc::MOP_DK, dk({0, 7, O | 11}, 16), 15 + 8 * entry);
            ok &= expect(false, "misaligned table", zc::MOP_DK, dk({0, 7, O | 11}, 8), 16 + 8 * entry);
            ok &= expect(false, "unknown kind", 9, ab(0, 1));
            if (!ok) return 1;
        }
    std::printf("ok operands: %d taken, %d refused\n", n_ok, n_bad);
    return 0;
}
