// CPU check of the rule that takes trajectories in sweeps (qgpu::traj_sweeps): never
// below 11 qubits (12 for merged blocks), where sweeps took up to twice the time;
// below the measured crossing of noise per step from there to 14; always above, where
// only tile passes hold sweeps. Built and run by tests/test_traj_form.py.
#include <cstdio>

#include "traj.hpp"

using namespace qgpu;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);                   \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

int main() {
    for (int n = 1; n <= 10; ++n)
        for (double p : {0.0, 1e-3, 0.5}) EXPECT(!traj_sweeps(n, p) && !traj_sweeps(n, p, true));
    EXPECT(!traj_sweeps(11, 0.0, true));
    for (int n = 12; n <= 14; ++n) EXPECT(traj_sweeps(n, 0.0, true));
    // gate by gate is the faster form at these, sweeps at those
    const double slow[4] = {0.005, 0.005, 0.015, 0.04}, fast[4] = {0.002, 0.002, 0.007, 0.015};
    for (int n = 11; n <= 14; ++n) {
        EXPECT(traj_sweeps(n, 0.0) && traj_sweeps(n, fast[n - 11]) && !traj_sweeps(n, slow[n - 11]));
        EXPECT(!traj_sweeps(n, 1.0));
    }
    for (int n = 15; n <= 20; ++n) EXPECT(traj_sweeps(n, 0.0) && traj_sweeps(n, 1.0));
    if (fails) return 1;
    std::printf("trajectory forms ok\n");
    return 0;
}
