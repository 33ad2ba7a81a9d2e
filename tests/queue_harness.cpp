// Host check of the op queue (OpQueue, plan_sweep from its head, consume_plan):
// the plans are those of a vector whose front is taken out, and the host cost
// per op does not grow with the length of the queue. Links the built
// libzeno_cuda.so; no GPU.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "zc_internal.h"

using zc::QOp;

static std::mt19937_64 rng(5);

// A random op; `dense` of 100 are two- or three-qubit blocks, 10 diagonals.
static QOp random_op(uint32_t n, int dense) {
    QOp op{};
    const int r = (int)(rng() % 100);
    auto support = [&](uint32_t k) {
        std::vector<uint32_t> all(n);
        for (uint32_t i = 0; i < n; i++) all[i] = i;
        std::shuffle(all.begin(), all.end(), rng);
        std::sort(all.begin(), all.begin() + k);
        op.k = k;
        for (uint32_t i = 0; i < k; i++) op.qs[i] = all[i];
    };
    if (r < dense || r >= 60) {
        op.kind = zc::Q_UNITARY;
        support(r < dense ? 2 + (uint32_t)(rng() % 2) : 1);
        op.data.assign((size_t)2 << (2 * op.k), 0.0);
        const double t = (double)(rng() % 1000) / 100.0;
        for (uint32_t j = 0; j < 1u << op.k; j++) op.data[2 * (j << op.k | j)] = 1.0;
        if (op.k == 1) {
            const double u[8] = {std::cos(t), 0, -std::sin(t), 0, std::sin(t), 0, std::cos(t), 0};
            op.data.assign(u, u + 8);
        }
    } else if (r < dense + 10) {
        op.kind = zc::Q_DIAG;
        support(1 + (uint32_t)(rng() % 3));
        for (uint32_t j = 0; j < 1u << op.k; j++) {
            const double t = (double)(rng() % 1000) / 100.0;
            op.data.push_back(std::cos(t));
            op.data.push_back(std::sin(t));
        }
    } else {
        op.kind = r % 5 ? zc::Q_CX : zc::Q_SWAP;
        op.a = (uint32_t)(rng() % n);
        do op.b = (uint32_t)(rng() % n);
        while (op.b == op.a);
    }
    return op;
}

static bool sweepable(const QOp &op) { return !(op.kind == zc::Q_UNITARY && op.k > 1); }
static bool same_op(const QOp &a, const QOp &b) {
    return a.kind == b.kind && a.k == b.k && !memcmp(a.qs, b.qs, sizeof a.qs) && a.a == b.a && a.b == b.b &&
           a.data == b.data;
}

// The flush loop on both kinds of queue, plan by plan.
static int same_plans(uint32_t n, int prec, bool ex, uint32_t L, uint32_t Hcap, size_t count, int dense) {
    std::vector<QOp> v;
    zc::OpQueue q;
    for (size_t i = 0; i < count; i++) {
        v.push_back(random_op(n, dense));
        q.push(QOp(v.back()));
    }
    while (!v.empty()) {
        if (q.size() != v.size()) return 1;
        for (size_t i = 0; i < std::min<size_t>(v.size(), 50); i++)
            if (!same_op(v[i], q[i])) return 2;
        zc::SweepPlan a, b;
        size_t na = 0, nb = 0;
        if (sweepable(v.front())) {
            na = zc::plan_sweep(n, prec, ex, L, Hcap, v, &a);
            nb = zc::plan_sweep(n, prec, ex, L, Hcap, q.ops, &b, q.head, q.touch);
        }
        if (na != nb) return 3;
        if (na <= 1) {
            v.erase(v.begin());
            q.pop();
            continue;
        }
        if (a.mops.size() != b.mops.size() || memcmp(a.mops.data(), b.mops.data(), a.mops.size() * sizeof(zc::MicroOp)) ||
            a.tables != b.tables || memcmp(&a.g, &b.g, sizeof a.g) || a.carry.size() != b.carry.size())
            return 4;
        zc::consume_plan(v, a);
        zc::consume_plan(q.ops, b, &q.head);
    }
    return q.empty() ? 0 : 5;
}

// Host time per op of the flush loop over `count` ops, us: dense two-qubit
// blocks and CX in turn, as a circuit fused to two qubits gives them.
static double cost(uint32_t n, size_t count) {
    double best = 1e30;
    for (int rep = 0; rep < 5; rep++) {
        zc::OpQueue q;
        for (size_t i = 0; i < count; i++) {
            QOp op = random_op(n, i % 2 ? 0 : 100);
            if (i % 2) {
                op = QOp{zc::Q_CX, 0, {}, (uint32_t)(rng() % n), 0, {}};
                op.b = (op.a + 1 + (uint32_t)(rng() % (n - 1))) % n;
            }
            q.push(std::move(op));
        }
        const auto t0 = std::chrono::steady_clock::now();
        while (!q.empty()) {
            zc::SweepPlan p;
            if (!sweepable(q.front()) || zc::plan_sweep(n, 64, false, 5, 3, q.ops, &p, q.head, q.touch) <= 1) q.pop();
            else zc::consume_plan(q.ops, p, &q.head);
        }
        const std::chrono::duration<double, std::micro> dt = std::chrono::steady_clock::now() - t0;
        best = std::min(best, dt.count() / (double)count);
    }
    return best;
}

int main() {
    for (int trial = 0; trial < 60; trial++) {
        const uint32_t n = 3 + (uint32_t)trial % 14, L = std::min<uint32_t>(n, 5), Hcap = std::min<uint32_t>(n - L, 7);
        const int mode = trial % 3, dense = trial % 4 == 3 ? 0 : 25;
        const int rc = same_plans(n, mode == 2 ? 32 : 64, mode == 0, L, trial % 2 ? Hcap : std::min<uint32_t>(Hcap, 2),
                                  trial % 5 == 0 ? 5000 : 300, dense);
        if (rc) return std::printf("FAIL trial %d: %d\n", trial, rc), 1;
    }
    const double few = cost(10, 250), many = cost(10, 8000);
    std::printf("ok plans; host us per op: %.3f of 250 ops, %.3f of 8000\n", few, many);
    return 0;
}
