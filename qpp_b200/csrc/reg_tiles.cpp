// reg_tiles.cpp -- host planning of the complex128 register tile passes
// (kernels_regtile.cu): which gates share a pass, and the program that moves
// their bits into place and applies them. No reference counterpart: Quantum++
// applies every gate as its own pass over the state (QEngine::visit_gate_step_,
// qengine.hpp:551-578 -> apply / applyCTRL).
#include "reg_tiles.hpp"

#include <algorithm>
#include <cstring>
#include <set>

namespace qgpu {

void reg_tile_shape(int nbits, int Tmax, int& T, int& L, int& NR) {
    T = std::max(kRtMinTile, std::min({nbits, Tmax, kRtMaxTile}));
    // Tiles of up to 2^11 amplitudes run 4 registers per thread (more warps,
    // fewer amplitudes each: few tiles, bound by latency), the full 2^12 tile
    // 16 (9 bits inside a warp, 8 warps).
    NR = T == kRtMaxTile ? 4 : 2;
    // runs of 2^L contiguous amplitudes; a tile keeps room for two targets
    L = T >= nbits ? T : std::min(4, T - 2);
}

static int target_bits(const GateDesc& g, int (&b)[2]) {
    b[0] = g.b0;
    b[1] = g.b1;
    return g.op == 2 ? 2 : 1;
}

std::vector<GateDesc> schedule_reg_gates(const std::vector<GateDesc>& gates, int nbits, int Tmax) {
    int T, L, NR;
    reg_tile_shape(nbits, Tmax, T, L, NR);
    return schedule_gates(gates, nbits, L, T - L, NR + 5);
}

namespace {

// Program bytes of one gate at most: two moves, a layout change with its two
// tables, the gate and its coefficients.
constexpr size_t kGateBytes[3] = {0, 3 * sizeof(RtOp) + 2 * sizeof(RtLayoutTab) + 64,
                                  4 * sizeof(RtOp) + 2 * sizeof(RtLayoutTab) + 512};

// One pass's program under construction.
struct Builder {
    int T, NR, inwarp;
    std::vector<RtOp> ops;
    std::vector<RtLayoutTab> lays;
    std::vector<cd> coef;
    int at[16]; // slot -> tile bit

    int slot_of(int bit) const { return int(std::find(at, at + T, bit) - at); }

    void table() {
        RtLayoutTab t;
        std::memset(&t, 0, sizeof(t));
        for (int s = 0; s < T; ++s) t.img[s] = uint16_t(rt_swz(1u << at[s]));
        lays.push_back(t);
    }

    RtOp& op(uint8_t type, int a = 0, int b = 0, uint32_t c = 0) {
        RtOp o;
        std::memset(&o, 0, sizeof(o));
        o.type = type;
        o.a = uint8_t(a);
        o.b = uint8_t(b);
        o.coef = c;
        ops.push_back(o);
        return ops.back();
    }

    // The layout for the gates [i, e) (their bits fit in a warp), `later` the
    // order in which the pass's other bits are wanted afterwards.
    void choose(const std::vector<GateDesc>& g, size_t i, size_t e, const std::vector<int>& later,
                bool first) {
        int use[16] = {0};
        std::vector<int> in; // bits of these gates
        int pair[2] = {-1, -1};
        for (size_t k = i; k < e; ++k) {
            int b[2];
            const int nb = target_bits(g[k], b);
            if (nb == 2 && pair[0] < 0) {
                pair[0] = b[0];
                pair[1] = b[1];
            }
            for (int x = 0; x < nb; ++x) {
                if (!use[b[x]]++) in.push_back(b[x]);
            }
        }
        for (int b : later)
            if (int(in.size()) < inwarp && std::find(in.begin(), in.end(), b) == in.end()) in.push_back(b);
        for (int b = 0; b < T && int(in.size()) < inwarp; ++b)
            if (std::find(in.begin(), in.end(), b) == in.end()) in.push_back(b);
        int next[16], n = 0;
        bool used[16] = {false};
        std::fill(next, next + 16, -1);
        // lane slots 0 and 1: the first 2-qubit gate's bits
        if (pair[0] < 0) { // none: the bits of the fewest gates
            std::vector<int> r = in;
            std::stable_sort(r.begin(), r.end(), [&](int x, int y) { return use[x] < use[y]; });
            pair[0] = r[0];
            pair[1] = r[1];
        }
        next[NR] = pair[0];
        next[NR + 1] = pair[1];
        used[pair[0]] = used[pair[1]] = true;
        // register slots: the most used of the others
        std::vector<int> rest;
        for (int b : in)
            if (!used[b]) rest.push_back(b);
        std::stable_sort(rest.begin(), rest.end(), [&](int x, int y) { return use[x] > use[y]; });
        for (int s = 0; s < NR; ++s) {
            next[s] = rest[size_t(n)];
            used[rest[size_t(n++)]] = true;
        }
        // lane slot 2: a bit whose shared-memory column differs from lane
        // slots 0 and 1 (element bits of one class modulo 3 share a column)
        std::vector<int> lanes(rest.begin() + n, rest.end());
        for (size_t x = 0; x < lanes.size(); ++x)
            if (lanes[x] % 3 != pair[0] % 3 && lanes[x] % 3 != pair[1] % 3) {
                std::swap(lanes[0], lanes[x]);
                break;
            }
        for (size_t x = 0; x < lanes.size(); ++x) {
            next[NR + 2 + int(x)] = lanes[x];
            used[lanes[x]] = true;
        }
        n = inwarp;
        for (int b = 0; b < T; ++b)
            if (!used[b]) next[n++] = b;
        if (first) {
            std::copy(next, next + T, at);
            table();
            return;
        }
        op(kRtLayout, 0, 0, uint32_t(lays.size()));
        table();
        std::copy(next, next + T, at);
        table();
    }

    // Brings both bits into lane slots 0 and 1.
    void to_pair(int p, int q) {
        int lane_of[2] = {at[NR], at[NR + 1]};
        bool free_slot[2];
        for (int x = 0; x < 2; ++x) free_slot[x] = lane_of[x] != p && lane_of[x] != q;
        int perm[5] = {0, 1, 2, 3, 4};
        bool permute = false;
        for (int bit : {p, q}) {
            const int s = slot_of(bit);
            if (s == NR || s == NR + 1) continue;
            const int x = free_slot[0] ? 0 : 1;
            free_slot[x] = false;
            if (s < NR) {
                op(kRtSwap, x, s);
                std::swap(at[NR + x], at[s]);
            } else {
                std::swap(perm[x], perm[s - NR]);
                permute = true;
            }
        }
        if (!permute) return;
        uint32_t c = 0;
        int old[5];
        std::copy(at + NR, at + NR + 5, old);
        for (int i = 0; i < 5; ++i) {
            c |= uint32_t(perm[i]) << (3 * i);
            at[NR + i] = old[perm[i]];
        }
        op(kRtPerm, 0, 0, c);
    }

    void gate(const GateDesc& g, const std::vector<std::pair<int, int>>& local,
              const std::vector<std::pair<int, int>>& outside) {
        RtOp o;
        std::memset(&o, 0, sizeof(o));
        if (g.op == 2) {
            to_pair(g.b0, g.b1);
            o.type = kRtG2;
        } else {
            const int s = slot_of(g.b0);
            o.type = s < NR ? kRtG1R : kRtG1L;
            o.a = uint8_t(s < NR ? s : s - NR);
        }
        o.coef = uint32_t(coef.size());
        o.ctrl = !local.empty() || !outside.empty();
        for (auto& c : local) {
            const int s = slot_of(c.first);
            uint8_t& m = s < NR ? o.rmask : s < NR + 5 ? o.lmask : o.wmask;
            uint8_t& v = s < NR ? o.rval : s < NR + 5 ? o.lval : o.wval;
            const int k = s < NR ? s : s < NR + 5 ? s - NR : s - NR - 5;
            m = uint8_t(m | (1u << k));
            if (c.second) v = uint8_t(v | (1u << k));
        }
        for (auto& c : outside) {
            o.gmask |= uint64_t(1) << c.first;
            if (c.second) o.gval |= uint64_t(1) << c.first;
        }
        ops.push_back(o);
        if (g.op == 1) {
            for (int r = 0; r < 2; ++r)
                for (int c = 0; c < 2; ++c) coef.push_back(g.A[r + 2 * c]);
            return;
        }
        // the matrix over the amplitude index lane & 3, as the fragments of a
        // real 4 x 8 matrix: lane l holds row k = l & 3, column l >> 2 = 2 j +
        // part of the products with real parts (x) and imaginary parts (y)
        auto row = [&](int k) {
            const int v0 = at[NR] == g.b0 ? k & 1 : k >> 1;
            const int v1 = at[NR] == g.b0 ? k >> 1 : k & 1;
            return 2 * v0 + v1;
        };
        for (int l = 0; l < 32; ++l) {
            const int k = l & 3, j = l >> 3, part = (l >> 2) & 1;
            const cd u = g.A[row(j) + 4 * row(k)];
            coef.push_back(part ? cd(u.imag(), u.real()) : cd(u.real(), -u.imag()));
        }
    }
};

} // namespace

void plan_reg_program(const std::vector<GateDesc>& gates, int nbits, int Tmax, RegProgram& P) {
    P.nbits = nbits;
    P.gates = gates;
    P.passes.clear();
    P.blob.clear();
    int T, L, NR;
    reg_tile_shape(nbits, Tmax, T, L, NR);
    const int nfree = T - L;
    for (size_t i = 0; i < gates.size();) {
        // the pass: gates in order while their bits above the low L fit
        uint64_t hi = 0;
        size_t j = i, bytes = 0;
        for (; j < gates.size(); ++j) {
            int b[2];
            const int nb = target_bits(gates[j], b);
            uint64_t h2 = hi;
            for (int x = 0; x < nb; ++x)
                if (b[x] >= L) h2 |= uint64_t(1) << b[x];
            bytes += kGateBytes[nb];
            if (__builtin_popcountll(h2) > nfree || bytes > kRtBlobMax) break;
            hi = h2;
        }
        if (j == i) raise(QGPU_ERR_NOT_SUPPORTED, "qgpu_run_gates()", "tile too small");
        // bits left over: the lowest others, for longer runs
        for (int b = L; __builtin_popcountll(hi) < nfree; ++b) hi |= uint64_t(1) << b;
        RegPass p;
        std::memset(&p, 0, sizeof(p));
        p.T = T;
        p.L = L;
        p.NR = NR;
        int nh = 0;
        for (int b = 0; b < 64; ++b)
            if ((hi >> b) & 1u) p.hi[nh++] = b;
        p.ntiles = nbits > T ? uint64_t(1) << (nbits - T) : 1;
        p.nvalid = nbits < T ? 1u << nbits : 1u << T;
        p.first = uint32_t(i);
        p.ngates = uint32_t(j - i);
        auto local = [&](int b) {
            return b < L ? b : L + int(std::find(p.hi, p.hi + nh, b) - p.hi);
        };
        // the gates on tile bits
        std::vector<GateDesc> g(gates.begin() + ptrdiff_t(i), gates.begin() + ptrdiff_t(j));
        for (GateDesc& x : g) {
            x.b0 = local(x.b0);
            if (x.op == 2) x.b1 = local(x.b1);
        }
        Builder B;
        B.T = T;
        B.NR = NR;
        B.inwarp = NR + 5;
        for (size_t k = 0; k < g.size();) {
            // the longest run whose bits fit in a warp
            uint32_t bits = 0;
            size_t e = k;
            for (; e < g.size(); ++e) {
                int b[2];
                const int nb = target_bits(g[e], b);
                uint32_t w = bits;
                for (int x = 0; x < nb; ++x) w |= 1u << b[x];
                if (__builtin_popcount(w) > B.inwarp) break;
                bits = w;
            }
            bool fits = k > 0;
            for (int s = B.inwarp; s < T && fits; ++s) fits = !((bits >> B.at[s]) & 1u);
            if (!fits) {
                std::vector<int> later;
                for (size_t x = e; x < g.size() && later.size() < 16; ++x) {
                    int b[2];
                    const int nb = target_bits(g[x], b);
                    for (int y = 0; y < nb; ++y)
                        if (std::find(later.begin(), later.end(), b[y]) == later.end()) later.push_back(b[y]);
                }
                B.choose(g, k, e, later, k == 0);
            }
            for (; k < e; ++k) {
                std::vector<std::pair<int, int>> in, out;
                for (auto& c : g[k].ctrl) {
                    const bool tile = c.first < L || ((hi >> c.first) & 1u);
                    if (tile) in.push_back({local(c.first), c.second});
                    else out.push_back(c);
                }
                B.gate(g[k], in, out);
            }
        }
        B.table();
        p.nops = uint32_t(B.ops.size());
        p.nlay = uint32_t(B.lays.size());
        p.blob = uint32_t(P.blob.size());
        const size_t b_ops = (B.ops.size() * sizeof(RtOp) + 15) / 16 * 16;
        const size_t b_lay = B.lays.size() * sizeof(RtLayoutTab);
        p.blob_bytes = uint32_t(b_ops + b_lay + B.coef.size() * sizeof(cd));
        P.blob.resize(P.blob.size() + p.blob_bytes);
        unsigned char* d = P.blob.data() + p.blob;
        std::memcpy(d, B.ops.data(), B.ops.size() * sizeof(RtOp));
        std::memcpy(d + b_ops, B.lays.data(), b_lay);
        std::memcpy(d + b_ops + b_lay, B.coef.data(), B.coef.size() * sizeof(cd));
        P.passes.push_back(p);
        i = j;
    }
}

} // namespace qgpu
