// CPU check of qgpu::fuse_wide: random circuits of gates, fan and controlled
// gates on 2-11 qubits, some with 3-qubit gates and steps that stay as they are;
// the blocks applied one by one must equal the dense steps applied one by one
// within 1e-12 (relative, max-norm), hold at most max_k qubits each, and keep
// every other step in its place. Built and run by tests/test_fuse_wide.py.
#include <algorithm>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

#include "circuit.hpp"

using namespace qgpu;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            if (fails < 20) std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);   \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

static void apply_dense(std::vector<cd>& psi, int n, const std::vector<int>& q, const std::vector<cd>& U) {
    const int k = int(q.size());
    const uint64_t D = uint64_t(1) << k;
    std::vector<uint64_t> off(D, 0);
    uint64_t mask = 0;
    for (int j = 0; j < k; ++j) {
        const uint64_t b = uint64_t(1) << (n - 1 - q[size_t(j)]);
        mask |= b;
        for (uint64_t i = 0; i < D; ++i)
            if ((i >> (k - 1 - j)) & 1u) off[i] |= b;
    }
    std::vector<cd> x(D);
    for (uint64_t r = 0; r < psi.size(); ++r) {
        if (r & mask) continue;
        for (uint64_t i = 0; i < D; ++i) x[i] = psi[r + off[i]];
        for (uint64_t i = 0; i < D; ++i) {
            cd s = 0;
            for (uint64_t j = 0; j < D; ++j) s += U[i + D * j] * x[j];
            psi[r + off[i]] = s;
        }
    }
}

int main() {
    std::mt19937_64 rng(17);
    std::normal_distribution<double> nd;
    int cases = 0;
    for (int n = 2; n <= 11; ++n)
        for (uint32_t max_k : {4u, 5u, 6u})
            for (int rep = 0; rep < 3; ++rep) {
                std::vector<Step> steps;
                std::vector<size_t> barriers;
                for (int k = 0; k < 40; ++k) {
                    std::vector<uint64_t> p(static_cast<size_t>(n));
                    for (int i = 0; i < n; ++i) p[size_t(i)] = uint64_t(i);
                    std::shuffle(p.begin(), p.end(), rng);
                    Step s;
                    const int kind = int(rng() % 12);
                    s.kind = StepKind::Gate;
                    if (kind == 0 && rep == 2) {
                        s.kind = StepKind::Nop;
                        barriers.push_back(steps.size());
                        steps.push_back(s);
                        continue;
                    }
                    if (kind < 5 || n < 3) s.target = {p[0]};
                    else if (kind < 8) s.target = {p[0], p[1]};
                    else if (kind < 9) s.target = {p[0], p[1], p[2]};
                    else if (kind < 11) s.kind = StepKind::Ctrl, s.ctrl = {p[1], p[2]}, s.target = {p[0]};
                    else s.kind = StepKind::Fan, s.target = {p[0], p[1]};
                    s.DU = s.kind == StepKind::Gate ? uint64_t(1) << s.target.size() : 2;
                    s.U.resize(s.DU * s.DU);
                    for (uint64_t r = 0; r < s.DU; ++r) { // rows of unit norm
                        double t = 0;
                        for (uint64_t c = 0; c < s.DU; ++c) t += std::norm(s.U[r + s.DU * c] = cd(nd(rng), nd(rng)));
                        for (uint64_t c = 0; c < s.DU; ++c) s.U[r + s.DU * c] /= std::sqrt(t);
                    }
                    steps.push_back(s);
                }
                std::vector<cd> a(size_t(1) << n), b;
                for (cd& x : a) x = cd(nd(rng), nd(rng));
                b = a;
                for (const Step& s : steps) {
                    std::vector<int> q;
                    std::vector<cd> U;
                    if (step_dense(s, 6, q, U)) apply_dense(a, n, q, U);
                }
                size_t at = 0;
                for (const Block& blk : fuse_wide(steps, uint32_t(n), max_k)) {
                    if (blk.step >= 0) {
                        EXPECT(at < barriers.size() && size_t(blk.step) == barriers[at]);
                        ++at;
                        continue;
                    }
                    EXPECT(!blk.qubits.empty() && blk.qubits.size() <= max_k);
                    EXPECT(blk.U.size() == size_t(1) << (2 * blk.qubits.size()));
                    apply_dense(b, n, blk.qubits, blk.U);
                }
                EXPECT(at == barriers.size());
                double err = 0, top = 0;
                for (size_t i = 0; i < a.size(); ++i) {
                    err = std::max(err, std::abs(a[i] - b[i]));
                    top = std::max(top, std::abs(a[i]));
                }
                EXPECT(err <= 1e-12 * top);
                ++cases;
            }
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("wide blocks ok: %d cases\n", cases);
    return 0;
}
