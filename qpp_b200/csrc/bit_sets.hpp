// bit_sets.hpp -- choosing the bits (qubits) that the next pass, warp stretch or
// fused block works on.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <utility>
#include <vector>

namespace qgpu {

// A gate waiting to be placed: its target bits and all its bits (targets and
// controls).
struct Waiting {
    uint64_t t, a;
    uint32_t id;
    uint32_t weight;
};

// The planners look at this many waiting gates at a time and take up the next
// ones as gates leave, so that a plan's cost grows with its gates and not with
// their square. A pass or block takes a few dozen gates, a full tile program up to
// 150.
constexpr size_t kLookAhead = 1024;

// At most kLookAhead waiting gates. The first ones are looked at one by one; beyond
// them, words of 64 gates with a mask of those that touch each bit.
class GateReach {
  public:
    explicit GateReach(const std::vector<Waiting>& gates) : g(gates), words((gates.size() + 63) / 64) {
        for (const Waiting& x : g) all_ |= x.a;
        if (words <= kScan) return;
        for (uint64_t m = all_; m; m &= m - 1)
            std::fill(touch[__builtin_ctzll(m)] + kScan, touch[__builtin_ctzll(m)] + words, uint64_t(0));
        for (size_t i = 64 * kScan; i < g.size(); ++i)
            for (uint64_t m = g[i].a; m; m &= m - 1) touch[__builtin_ctzll(m)][i / 64] |= uint64_t(1) << (i % 64);
    }

    // The union of the gates' bits.
    uint64_t all() const { return all_; }

    // The gates that a set of bits S can take: in order, every gate whose targets
    // lie in S and which shares no bit with an earlier gate left behind. Their
    // weights' sum. A gate that runs has all its targets among the bits of S with
    // nothing left behind on them (live), so the sum ends with the last such bit, and
    // beyond the first gates only those that touch one are looked at: a bit of S
    // whose next gate is far away costs no scan up to it.
    uint32_t operator()(uint64_t S) const {
        const uint64_t in = S & all_;
        uint64_t behind = 0;
        uint32_t sum = 0;
        for (const Waiting *x = g.data(), *const end = x + std::min(g.size(), 64 * kScan); x != end; ++x) {
            if (!(x->t & ~S) && !(x->a & behind)) {
                sum += x->weight;
            } else {
                behind |= x->a;
                if (!(in & ~behind)) return sum;
            }
        }
        return words <= kScan ? sum : sum + beyond(S, behind);
    }

  private:
    static constexpr size_t kScan = 2; // words looked at one by one
    // The sum over the words from kScan on, `behind` left there by the gates before.
    __attribute__((noinline)) uint32_t beyond(uint64_t S, uint64_t behind) const {
        uint64_t live = S & all_ & ~behind;
        uint64_t ran[kLookAhead / 64];
        uint32_t sum = 0;
        for (size_t w = kScan; w < words && live; ++w) {
            uint64_t m = at(live, w);
            ran[w] = 0;
            while (m) {
                const uint64_t bit = m & (0 - m);
                const Waiting& x = g[w * 64 + size_t(__builtin_ctzll(m))];
                m ^= bit;
                if (!(x.t & ~S) && !(x.a & behind) &&
                    (!(x.a & ~S) || free_of(x.a & ~S, ran, w, bit))) {
                    sum += x.weight;
                    ran[w] |= bit;
                    continue;
                }
                behind |= x.a & S;
                if (!(live & x.a)) continue;
                live &= ~x.a;
                m &= at(live, w);
            }
        }
        return sum;
    }
    // The gates of word w that touch a bit of `bits`.
    uint64_t at(uint64_t bits, size_t w) const {
        uint64_t m = 0;
        for (; bits; bits &= bits - 1) m |= touch[__builtin_ctzll(bits)][w];
        return m;
    }
    // Whether every gate from word kScan on and before gate `bit` of word w that
    // touches one of `bits` (controls outside the set) has run.
    bool free_of(uint64_t bits, const uint64_t* ran, size_t w, uint64_t bit) const {
        for (; bits; bits &= bits - 1) {
            const uint64_t* const t = touch[__builtin_ctzll(bits)];
            uint64_t left = t[w] & ~ran[w] & (bit - 1);
            for (size_t v = kScan; v < w; ++v) left |= t[v] & ~ran[v];
            if (left) return false;
        }
        return true;
    }
    const std::vector<Waiting>& g;
    const size_t words;
    uint64_t all_ = 0;
    uint64_t touch[64][kLookAhead / 64]; // rows of all_, words from kScan on
};

// The set of `size` bits (those of `fixed` among them, out of `pool`) whose
// reach is large: grown from the first gate (grow: by the gate whose new bits
// raise the reach the most per bit; else in gate order), then improved by
// trading one bit at a time. Trading costs the bits in times the bits out
// evaluations, growing one for every different set of targets. 12000 2-qubit gates
// on 28 qubits plan in 0.04 s as passes and 0.3 s as blocks of 6, also with a qubit
// that idles until the last gate (1.2 s and two minutes for 10000 when every
// evaluation looked at all remaining gates).
inline uint64_t choose_bits(const std::vector<Waiting>& g, uint64_t fixed, uint64_t pool, int size,
                            bool grow = false) {
    const GateReach reach(g);
    const uint64_t all = reach.all();
    uint64_t S = fixed, behind = 0;
    if (grow) {
        // the different target sets, in the order they first appear, until every
        // bit has been met
        std::vector<uint64_t> sets;
        for (const Waiting& x : g) {
            sets.push_back(x.t);
            if ((behind |= x.t) == all) break;
        }
        if (sets.size() > 64) { // below, evaluating some twice costs less than this
            std::vector<std::pair<uint64_t, size_t>> first(sets.size());
            for (size_t i = 0; i < sets.size(); ++i) first[i] = {sets[i], i};
            std::sort(first.begin(), first.end());
            std::vector<size_t> keep;
            for (size_t i = 0; i < first.size(); ++i)
                if (i == 0 || first[i].first != first[i - 1].first) keep.push_back(first[i].second);
            std::sort(keep.begin(), keep.end());
            for (size_t i = 0; i < keep.size(); ++i) sets[i] = sets[keep[i]];
            sets.resize(keep.size());
        }
        if (!g.empty() && __builtin_popcountll(S | g[0].t) <= size) S |= g[0].t;
        while (__builtin_popcountll(S) < size) {
            const uint32_t r0 = reach(S);
            uint64_t top = 0;
            double best = -1;
            for (uint64_t t : sets) {
                const int add = __builtin_popcountll(t & ~S);
                if (add && __builtin_popcountll(S) + add <= size) {
                    const double q = double(reach(S | t) - r0) / add;
                    if (q > best) {
                        best = q;
                        top = S | t;
                    }
                }
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
    uint32_t best = reach(S);
    for (int round = 0; round < 8; ++round) {
        uint64_t top = S;
        for (uint64_t in = S & ~fixed; in; in &= in - 1)
            for (uint64_t out = pool & all & ~S; out; out &= out - 1) {
                const uint64_t S2 = (S ^ (in & (0 - in))) | (out & (0 - out));
                const uint32_t r = reach(S2);
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
