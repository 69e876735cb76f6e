// CPU check of SegPlan's 32-bit digits (qgpu::seg_magic, qgpu::seg_offset): for
// random plans and for every divisor up to 3000 and a spread of larger ones with
// counts just below 2^31, the offsets of the first and last group numbers, of the
// ends of digits and of random ones must equal those of the 64-bit divisions.
// Built and run by tests/test_seg_plan.py.
#include <cstdio>
#include <cstring>
#include <random>

#include "kernels.hpp"

using namespace qgpu;

static long bad = 0, tried = 0;

static void compare(SegPlan p, uint64_t g) {
    if (g >= p.count) return;
    p.pow2 = 0;
    p.small = 1;
    SegPlan q = p;
    q.small = 0;
    bad += seg_offset(p, g) != seg_offset(q, g);
    ++tried;
}

int main() {
    std::mt19937_64 rng(1);
    for (int rep = 0; rep < 3000; ++rep) {
        SegPlan p;
        std::memset(&p, 0, sizeof(p));
        p.count = 1;
        p.fixed_off = rng() % 1000;
        while (p.nseg < 12) {
            const uint64_t d = 2 + rng() % (rep % 3 ? 9 : 5000);
            if (p.count * d >= uint64_t(1) << 31) break;
            p.size[p.nseg] = d;
            p.stride[p.nseg++] = rng() % 1000000007;
            p.count *= d;
            if (rng() % 9 == 0) break;
        }
        seg_magic(p);
        for (uint64_t k = 0; k < 50; ++k) {
            compare(p, k);
            compare(p, p.count - 1 - k);
            compare(p, rng() % p.count);
        }
    }
    for (uint64_t d = 2; d < 1000000000; d = d < 3000 ? d + 1 : d * 5 / 4 + 1) {
        SegPlan p;
        std::memset(&p, 0, sizeof(p));
        p.nseg = 2;
        p.size[0] = d;
        p.size[1] = ((uint64_t(1) << 31) - 1) / d;
        p.stride[0] = 1;
        p.stride[1] = uint64_t(1) << 33;
        p.count = p.size[0] * p.size[1];
        if (p.size[1] < 2) break;
        seg_magic(p);
        if (!p.small) ++bad;
        for (uint64_t k = 0; k < 100; ++k) {
            const uint64_t row = rng() % p.size[1] * d;
            compare(p, k);
            compare(p, p.count - 1 - k);
            compare(p, row);
            compare(p, row + d - 1);
        }
    }
    SegPlan big;
    std::memset(&big, 0, sizeof(big));
    big.nseg = 1;
    big.size[0] = big.count = uint64_t(1) << 31 | 1;
    seg_magic(big);
    bad += big.small; // 2^31 and more stay with 64 bits
    if (bad || tried < 100000) {
        std::printf("%ld failures of %ld\n", bad, tried);
        return 1;
    }
    std::printf("seg plan ok: %ld offsets\n", tried);
    return 0;
}
