// CPU check that a complex64 tile program planned `ordered`, which may trade registers
// as the kernels do not, is refused before anything reaches the device, while the plain
// one of the same gates is not marked. Built and run by tests/test_ordered_program.py.
#include <cstdio>

#include "internal.hpp"
#include "reg_tiles.hpp"

using namespace qgpu;

int main() {
    std::vector<GateDesc> g;
    for (int k = 0; k < 8; ++k) {
        GateDesc d;
        d.op = 2;
        d.b0 = k % 5;
        d.b1 = (k + 1) % 5;
        for (int i = 0; i < 16; ++i) d.A[i] = i % 5 ? 0.0 : 1.0;
        g.push_back(d);
    }
    RegProgram plain, ordered;
    plain.prec = ordered.prec = QGPU_C64;
    plan_reg_program(g, 14, 12, plain);
    plan_reg_program(g, 14, 12, ordered, nullptr, true);
    if (plain.trades || !ordered.trades) return std::printf("FAIL marks\n"), 1;
    qgpu_state s; // no context: nothing may be enqueued
    s.prec = QGPU_C64;
    s.dims.assign(14, 2);
    try {
        run_reg_program(&s, ordered);
    } catch (const Exc& e) {
        if (e.code != QGPU_ERR_NOT_SUPPORTED) return std::printf("FAIL code %d\n", int(e.code)), 1;
        std::printf("ordered program refused\n");
        return 0;
    }
    std::printf("FAIL not refused\n");
    return 1;
}
