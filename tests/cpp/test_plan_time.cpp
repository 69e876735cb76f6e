// CPU check of the look-ahead of the pass and block planners (qgpu::choose_bits,
// plan_reg_program, fuse_wide): GateReach against its definition over random gates
// with controls; circuits of 12000 gates in which every qubit is busy, one idles
// until the last gate, or the gates move along the register, planned within 1 s
// (passes) and 2 s (blocks), several times what they take (0.04 and 0.3 s); looking
// at all remaining gates for every set of bits took over 1.2 and 120 s where a
// qubit idles. And no more passes and blocks than an unlimited look-ahead finds.
// Built and run by tests/test_plan_time.py.
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

#include "bit_sets.hpp"
#include "circuit.hpp"
#include "reg_tiles.hpp"

using namespace qgpu;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            if (fails < 20) std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);   \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

// the weights that S can take, by the definition
static uint32_t reach_of(const std::vector<Waiting>& g, uint64_t S) {
    uint64_t behind = 0;
    uint32_t sum = 0;
    for (const Waiting& x : g) {
        if (!(x.t & ~S) && !(x.a & behind)) sum += x.weight;
        else behind |= x.a;
    }
    return sum;
}

static GateDesc gate2(int a, int b) {
    GateDesc g;
    g.op = 2;
    g.b0 = a;
    g.b1 = b;
    for (int i = 0; i < 16; ++i) g.A[i] = i % 5 ? 0.0 : 1.0;
    return g;
}

static Step step2(int a, int b) {
    Step s;
    s.kind = StepKind::Gate;
    s.target = {uint64_t(a), uint64_t(b)};
    s.DU = 4;
    s.U.assign(16, cd(0));
    for (int i = 0; i < 4; ++i) s.U[size_t(5 * i)] = 1.0;
    return s;
}

using Pair = std::pair<int, int>;

static double seconds_of(const std::vector<Pair>& g, int n, qgpu_prec prec, size_t& passes) {
    std::vector<GateDesc> d;
    for (const Pair& p : g) d.push_back(gate2(p.first, p.second));
    RegProgram P;
    P.prec = prec;
    const auto t0 = std::chrono::steady_clock::now();
    plan_reg_program(d, n, 12, P);
    passes = P.passes.size();
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

static double seconds_wide(const std::vector<Pair>& g, int n, size_t& blocks) {
    std::vector<Step> s;
    for (const Pair& p : g) s.push_back(step2(p.first, p.second));
    const auto t0 = std::chrono::steady_clock::now();
    const std::vector<Block> b = fuse_wide(s, uint32_t(n), 6);
    blocks = b.size();
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

int main() {
    std::mt19937 rng(5);
    auto pick = [&](int n) { return int(rng() % uint32_t(n)); };
    for (int rep = 0; rep < 300; ++rep) {
        const int n = 3 + pick(30);
        std::vector<Waiting> g;
        const int ng = 1 + pick(600);
        for (int k = 0; k < ng; ++k) {
            Waiting w{};
            w.t = uint64_t(1) << pick(n);
            if (pick(2)) w.t |= uint64_t(1) << pick(n);
            w.a = w.t;
            for (int c = pick(4) ? 0 : 1 + pick(2); c > 0; --c) w.a |= uint64_t(1) << pick(n);
            w.id = uint32_t(k);
            w.weight = 1 + uint32_t(pick(2));
            g.push_back(w);
        }
        const GateReach r(g);
        for (int q = 0; q < 40; ++q) {
            uint64_t S = 0;
            for (int c = pick(n); c >= 0; --c) S |= uint64_t(1) << pick(n);
            EXPECT(r(S) == reach_of(g, S));
        }
    }
    // circuits of 12000 gates
    const int n = 28, ng = 12000;
    std::vector<Pair> busy, idle, window;
    auto two = [&](int lo, int m) {
        const int a = pick(m);
        int b = pick(m - 1);
        b += b >= a;
        return Pair{lo + a, lo + b};
    };
    for (int k = 0; k < ng; ++k) {
        busy.push_back(two(0, n));
        idle.push_back(k + 1 < ng ? two(0, n - 1) : Pair{0, n - 1});
        window.push_back(two(k * (n - 8) / ng, 8));
    }
    for (const auto* c : {&busy, &idle, &window}) {
        size_t p;
        for (qgpu_prec prec : {QGPU_C128, QGPU_C64}) {
            const double s = seconds_of(*c, n, prec, p);
            std::printf("passes %zu in %.3f s\n", p, s);
            EXPECT(s < 1.0);
        }
        const double s = seconds_wide(*c, n, p);
        std::printf("blocks %zu in %.3f s\n", p, s);
        EXPECT(s < 2.0);
    }
    // layers of 2-qubit gates on a random matching; the counts of an unlimited
    // look-ahead
    struct Known {
        int n, layers;
        size_t passes, blocks;
    };
    const Known known[] = {{16, 8, 4, 11}, {20, 40, 30, 71}, {28, 12, 18, 32}, {30, 60, 92, 163}};
    for (const Known& w : known) {
        std::mt19937 r2(uint32_t(w.n));
        std::vector<Pair> c;
        for (int l = 0; l < w.layers; ++l) {
            std::vector<int> q;
            for (int i = 0; i < w.n; ++i) q.insert(q.begin() + int(r2() % uint32_t(i + 1)), i);
            for (int i = 0; i + 1 < w.n; i += 2) c.push_back({q[size_t(i)], q[size_t(i + 1)]});
        }
        size_t passes, blocks;
        seconds_of(c, w.n, QGPU_C128, passes);
        seconds_wide(c, w.n, blocks);
        std::printf("%d qubits, %d layers: %zu passes, %zu blocks\n", w.n, w.layers, passes, blocks);
        EXPECT(passes <= w.passes && blocks <= w.blocks);
    }
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("planning ok\n");
    return 0;
}
