// bit_sets.hpp -- choosing the bits (qubits) that the next pass, warp stretch or
// fused block works on.
#pragma once

#include <cstdint>
#include <vector>

namespace qgpu {

// A gate waiting to be placed: its target bits and all its bits (targets and
// controls).
struct Waiting {
    uint64_t t, a;
    uint32_t id;
    uint32_t weight;
};

// The gates that a set of bits S can take: in order, every gate whose targets
// lie in S and which shares no bit with an earlier gate left behind. Their
// weights' sum; `all`: the union of the gates' bits.
inline uint32_t reach(const std::vector<Waiting>& g, uint64_t S, uint64_t all) {
    uint64_t behind = 0;
    uint32_t sum = 0;
    for (const Waiting& x : g) {
        if (!(x.t & ~S) && !(x.a & behind)) {
            sum += x.weight;
        } else {
            behind |= x.a;
            if (behind == all) break;
        }
    }
    return sum;
}

// The set of `size` bits (those of `fixed` among them, out of `pool`) whose
// reach is large: grown from the first gate (grow: by the gate whose new bits
// raise the reach the most per bit; else in gate order), then improved by
// trading one bit at a time. Trading costs the bits in times the bits out
// evaluations of a few dozen gates each.
inline uint64_t choose_bits(const std::vector<Waiting>& g, uint64_t fixed, uint64_t pool, int size,
                            bool grow = false) {
    uint64_t all = 0, S = fixed, behind = 0;
    for (const Waiting& x : g) all |= x.a;
    if (grow) {
        if (!g.empty() && __builtin_popcountll(S | g[0].t) <= size) S |= g[0].t;
        while (__builtin_popcountll(S) < size) {
            const uint32_t r0 = reach(g, S, all);
            uint64_t top = 0;
            double best = -1;
            behind = 0;
            for (const Waiting& x : g) {
                const int add = __builtin_popcountll(x.t & ~S);
                if (add && __builtin_popcountll(S) + add <= size) {
                    const double q = double(reach(g, S | x.t, all) - r0) / add;
                    if (q > best) {
                        best = q;
                        top = S | x.t;
                    }
                }
                if ((behind |= x.t) == all) break;
            }
            if (!top) break;
            S = top;
        }
    } else {
        for (const Waiting& x : g) {
            if (!(x.a & behind) && __builtin_popcountll(S | x.t) <= size) S |= x.t;
            else if ((behind |= x.a) == all) break;
        }
    }
    for (uint64_t r = pool & ~S; r && __builtin_popcountll(S) < size; r &= r - 1) S |= r & (0 - r);
    uint32_t best = reach(g, S, all);
    for (int round = 0; round < 8; ++round) {
        uint64_t top = S;
        for (uint64_t in = S & ~fixed; in; in &= in - 1)
            for (uint64_t out = pool & all & ~S; out; out &= out - 1) {
                const uint64_t S2 = (S ^ (in & (0 - in))) | (out & (0 - out));
                const uint32_t r = reach(g, S2, all);
                if (r > best) {
                    best = r;
                    top = S2;
                }
            }
        if (top == S) break;
        S = top;
    }
    return S;
}

} // namespace qgpu
