// CPU check of the choice between the two fused plans (qgpu::fuse_best): planned without
// matrices, both have the blocks that they have with them; and the one taken is never
// the one with more passes of 3 to 6 qubits on 13 and more bits, while short circuits,
// where both need as many, take the greedy one with its smaller blocks. Random circuits of gates, fan
// and controlled gates, some of seven qubits, which stay as they are. Built and run by
// tests/test_fuse_best.py.
#include <algorithm>
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

static bool same(const std::vector<Block>& a, const std::vector<Block>& b, bool matrices) {
    if (a.size() != b.size()) return false;
    for (size_t i = 0; i < a.size(); ++i)
        if (a[i].step != b[i].step || a[i].qubits != b[i].qubits || (matrices && a[i].U != b[i].U)) return false;
    return true;
}

int main() {
    std::mt19937 rng(11);
    int wide = 0, greedy = 0;
    for (int n : {7, 9, 12, 13, 16, 24})
        for (int ng : {4, 10, 30, 80})
            for (int rep = 0; rep < 4; ++rep) {
                std::vector<Step> steps;
                for (int k = 0; k < ng; ++k) {
                    std::vector<uint64_t> p(static_cast<size_t>(n));
                    for (int i = 0; i < n; ++i) p[size_t(i)] = uint64_t(i);
                    for (size_t i = p.size(); i > 1; --i) std::swap(p[i - 1], p[rng() % i]);
                    Step s;
                    const int kind = int(rng() % 12);
                    s.kind = StepKind::Gate;
                    if (kind < 6) s.target = {p[0]};
                    else if (kind < 9) s.target = {p[0], p[1]};
                    else if (kind == 9) s.kind = StepKind::Ctrl, s.ctrl = {p[1], p[2]}, s.target = {p[0]};
                    else if (kind == 10) s.kind = StepKind::Fan, s.target = {p[0], p[1]};
                    else if (rep == 3) s.kind = StepKind::Ctrl, s.ctrl.assign(p.begin() + 1, p.begin() + 7), s.target = {p[0]};
                    else s.target = {p[0], p[1], p[2]};
                    s.DU = s.kind == StepKind::Gate ? uint64_t(1) << s.target.size() : 2;
                    s.U.assign(s.DU * s.DU, cd(0));
                    for (uint64_t r = 0; r < s.DU; ++r) s.U[r * (s.DU + 1)] = cd(0.6, 0.8);
                    steps.push_back(s);
                }
                const auto g = fuse(steps, uint32_t(n), 6), w = fuse_wide(steps, uint32_t(n), 6);
                EXPECT(same(g, fuse(steps, uint32_t(n), 6, true), false));
                EXPECT(same(w, fuse_wide(steps, uint32_t(n), 6, true), false));
                const auto best = fuse_best(steps, uint32_t(n), 6);
                const bool is_w = same(best, w, true), is_g = same(best, g, true);
                EXPECT(is_w || is_g);
                if (is_w && !is_g) ++wide;
                if (is_g && !is_w) ++greedy;
                // below 20 passes no difference of the small blocks' cost outweighs one
                if (n >= 13 && std::max(g.size(), w.size()) < 20)
                    EXPECT(best.size() == std::min(g.size(), w.size()));
                EXPECT(same(fuse_best(steps, uint32_t(n), 2), fuse(steps, uint32_t(n), 2), true));
            }
    EXPECT(wide > 10 && greedy > 5);
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("best blocks ok: %d wide, %d greedy\n", wide, greedy);
    return 0;
}
