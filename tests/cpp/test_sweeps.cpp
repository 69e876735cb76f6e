// CPU check of the trajectory kernel's sweeps (qgpu::plan_sweeps and
// qgpu::noise_steps): random programs of G1, CG1, G2, G3 gates and measurements
// on 4-18 qubits, tiled above 14. The instructions must come out in order and
// unchanged but for their slots; every sweep's bits must be four distinct ones of
// its register or tile, hold its gates' targets in the slots the flags name (a
// 2-qubit gate's b1 below its b0), and count its instructions and steps; a tile
// pass must count its headers; the noise steps must list the untiled index and
// the living qubits of every step. Built and run by tests/test_sweeps.py.
#include <cstdio>
#include <random>
#include <vector>

#include "traj.hpp"

using namespace qgpu;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            if (fails < 20) std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);   \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

int main() {
    std::mt19937 rng(3);
    int cases = 0, in_sweeps = 0, patterns = 0;
    for (int n = 3; n <= 18; ++n)
        for (int rep = 0; rep < 8; ++rep) {
            TProgram P;
            P.n = uint32_t(n);
            P.mats.assign(512, 0.f);
            for (int k = 0; k < 150; ++k) {
                int b[4];
                for (int i = 0; i < 4; ++i)
                    do {
                        b[i] = int(rng() % uint32_t(n));
                        for (int j = 0; j < i; ++j)
                            if (b[j] == b[i] && n > 3) b[i] = -1;
                    } while (b[i] < 0);
                TInstr I{};
                const int kind = int(rng() % 20);
                I.b0 = uint8_t(b[0]);
                I.flags = rng() % 4 ? kTNewStep : 0;
                I.mat = 2 * (rng() % 100);
                if (n == 3 || kind < 9) I.op = kTG1;
                else if (kind < 15) I.op = kTG2, I.b1 = uint8_t(b[1]);
                else if (kind < 17) I.op = kTCG1, I.cmask = 1u << b[1] | 1u << b[2], I.cval = rng() % 2 << b[1];
                else if (kind < 18) I.op = kTG3, I.b1 = uint8_t(b[1]), I.cmask = uint32_t(b[2]);
                else I.op = kTMeas, I.flags |= rng() % 3 ? 0 : kTDestructive;
                P.ins.push_back(I);
            }
            plan_tiles(P, rep % 2 ? 10 : 12);
            const TProgram before = P;
            plan_sweeps(P);
            std::vector<TInstr> flat;
            size_t tile_end = 0;
            int bits_here = n;
            for (size_t i = 0; i < P.ins.size(); ++i) {
                const TInstr& I = P.ins[i];
                if (i >= tile_end) bits_here = n;
                if (I.op == kTTile) {
                    tile_end = i + 1 + I.cmask;
                    bits_here = I.b0;
                    uint32_t gates = 0;
                    for (size_t k = i + 1; k < tile_end; ++k) gates += P.ins[k].op != kTSweep;
                    TInstr H = I;
                    H.cmask = gates;
                    flat.push_back(H);
                } else if (I.op == kTSweep) {
                    EXPECT(n > 14 ? i < tile_end : n >= 4);
                    uint32_t seen = 0, steps = 0;
                    for (int s = 0; s < 4; ++s) {
                        const uint32_t b = I.mat >> (8 * s) & 255u;
                        EXPECT(int(b) < bits_here && !(seen >> b & 1u));
                        seen |= 1u << b;
                    }
                    EXPECT(I.cmask >= 1 && I.cmask <= 24 && i + I.cmask < P.ins.size());
                    for (size_t k = i + 1; k <= i + I.cmask; ++k) {
                        const TInstr& G = P.ins[k];
                        const int a = G.flags >> 2 & 3, b = G.flags >> 4 & 3;
                        EXPECT(G.op == kTG1 || G.op == kTCG1 || G.op == kTG2);
                        EXPECT((I.mat >> (8 * a) & 255u) == (G.op == kTG2 ? G.b1 : G.b0));
                        if (G.op == kTG2) EXPECT(a < b && (I.mat >> (8 * b) & 255u) == G.b0);
                        steps += G.flags & kTNewStep;
                        ++in_sweeps;
                    }
                    EXPECT(steps == I.cval);
                    for (uint32_t k = 1; k <= I.cmask && I.b1 != kSweepAny; ++k) {
                        const TInstr& G = P.ins[i + k];
                        const int a = G.flags >> 2 & 3, b = G.flags >> 4 & 3;
                        if (I.b1 == kSweep4x1q) EXPECT(I.cmask == 4 && G.op == kTG1 && a == int(k) - 1);
                        else EXPECT(I.cmask == 2 && G.op == kTG2 && a == 2 * int(k) - 2 && b == a + 1);
                        ++patterns;
                    }
                } else {
                    flat.push_back(I);
                    flat.back().flags &= kTNewStep | kTDestructive;
                }
            }
            EXPECT(flat.size() == before.ins.size());
            for (size_t i = 0; i < flat.size() && i < before.ins.size(); ++i) {
                const TInstr &a = flat[i], &b = before.ins[i];
                EXPECT(a.op == b.op && a.b0 == b.b0 && a.b1 == b.b1 && a.flags == b.flags && a.mat == b.mat &&
                       a.cmask == b.cmask && a.cval == b.cval);
            }
            const std::vector<uint2> ns = noise_steps(P);
            size_t at = 0;
            uint32_t alive = (1u << n) - 1, orig = 0;
            for (const TInstr& I : before.ins) {
                if (I.op == kTTile) continue;
                if (I.flags & kTNewStep) {
                    EXPECT(at < ns.size() && ns[at].x == orig && ns[at].y == alive);
                    ++at;
                }
                if (I.op == kTMeas && (I.flags & kTDestructive)) alive &= ~(1u << I.b0);
                ++orig;
            }
            EXPECT(at == ns.size());
            ++cases;
        }
    EXPECT(in_sweeps > 1000 && patterns > 50);
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("sweeps ok: %d cases\n", cases);
    return 0;
}
