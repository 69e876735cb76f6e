// CPU check of the choice between the register QFT passes and the smaller tiles
// (qgpu::qft_reg_pays) on the planned pass counts: the smaller tiles at 30 forward
// complex64 targets with the reversal, in as many passes with groups no fuller; the
// register passes everywhere else, at 31 and 32 targets and at 33 and more, where they
// save a pass, as well. Built and run by tests/test_qft_choice.py.
#include <cstdio>
#include <numeric>
#include <vector>

#include "kernels.hpp"

using namespace qgpu;

int main() {
    int fails = 0;
    for (qgpu_prec prec : {QGPU_C128, QGPU_C64})
        for (int n = 13; n <= 36; ++n)
            for (int mode = 0; mode < 4; ++mode) {
                const bool inverse = mode & 1, rev = mode & 2;
                std::vector<uint64_t> t(static_cast<size_t>(n));
                std::iota(t.begin(), t.end(), 0);
                QftRegSchedule R;
                QftSchedule S;
                const uint64_t D = uint64_t(1) << n;
                if (!plan_qft_reg(prec, D, t, inverse, rev, R)) continue;
                if (!plan_qft(false, D, 2, prec == QGPU_C128 ? 16 : 8, t, inverse, rev, S)) continue;
                const bool pays = qft_reg_pays(prec, t.size(), R.plans.size(), rev, inverse);
                const bool want = !(prec == QGPU_C64 && rev && !inverse && n == 30);
                if (pays != want) {
                    std::printf("FAIL prec %d, %d qubits, inverse %d, reversal %d: %zu register passes, %zu smaller\n",
                                int(prec), n, int(inverse), int(rev), R.plans.size(), S.plans.size());
                    ++fails;
                }
                if (n >= 33 && R.plans.size() >= S.plans.size()) ++fails;
            }
    if (fails) return 1;
    std::printf("choice ok\n");
    return 0;
}
