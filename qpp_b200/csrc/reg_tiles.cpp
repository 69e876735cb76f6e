// reg_tiles.cpp -- host planning of the register tile passes
// (kernels_regtile.cu, kernels_regtile32.cu): which gates share a pass, and the
// program that moves their bits into place and applies them. No reference counterpart: Quantum++
// applies every gate as its own pass over the state (QEngine::visit_gate_step_,
// qengine.hpp:551-578 -> apply / applyCTRL).
#include "reg_tiles.hpp"

#include "bit_sets.hpp"

#include <algorithm>
#include <complex>
#include <cstring>

namespace qgpu {

void reg_tile_shape(qgpu_prec prec, int nbits, int Tmax, int& T, int& L, int& NR) {
    T = std::max(kRtMinTile, std::min({nbits, Tmax, kRtMaxTile}));
    // Tiles of up to 2^11 amplitudes run 4 registers per thread (more warps,
    // fewer amplitudes each: few tiles, bound by latency), the full 2^12 tile
    // 16 (9 bits inside a warp, 8 warps).
    NR = T == kRtMaxTile ? 4 : 2;
    // Runs of 2^L contiguous amplitudes (128 bytes, one line) leave 9 bits to
    // choose; L = 4 ran as fast (42.6 and 43.2 ms for 126 gates on 28 qubits)
    // with a few passes more. A tile keeps room for two targets.
    L = T >= nbits ? T : std::min(prec == QGPU_C128 ? 3 : 4, T - 2);
}

namespace {

// Program bytes of one gate at most: two moves, a layout change with its two
// tables, the gate and its coefficients.
constexpr size_t kGateBytes[3] = {0, 3 * sizeof(RtOp) + 2 * sizeof(RtLayoutTab) + 64,
                                  4 * sizeof(RtOp) + 2 * sizeof(RtLayoutTab) + 512};

// Moves the gates that S reaches from g to `out`, in order, at most `most`
// program bytes of them.
void take(std::vector<Waiting>& g, uint64_t S, size_t most, std::vector<Waiting>& out) {
    uint64_t behind = 0;
    size_t bytes = 0, keep = 0;
    bool full = false;
    for (const Waiting& x : g) {
        const size_t cost = kGateBytes[x.t & (x.t - 1) ? 2 : 1];
        if (!full && !(x.t & ~S) && !(x.a & behind) && bytes + cost <= most) {
            bytes += cost;
            out.push_back(x);
        } else {
            full = full || bytes + cost > most;
            behind |= x.a;
            g[keep++] = x;
        }
    }
    g.resize(keep);
}

// One pass's program under construction.
struct Builder {
    bool f32, ordered;
    int T, NR, inwarp;
    std::vector<RtOp> ops;
    std::vector<RtLayoutTab> lays;
    std::vector<cd> coef;
    std::vector<std::complex<float>> coef32;
    int at[16]; // slot -> tile bit

    int slot_of(int bit) const { return int(std::find(at, at + T, bit) - at); }

    void table() {
        RtLayoutTab t;
        std::memset(&t, 0, sizeof(t));
        for (int s = 0; s < T; ++s)
            t.img[s] = uint16_t(f32 ? rt_swz32(1u << at[s]) : rt_swz(1u << at[s]));
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

    // The layout for a stretch of gates inside the bits `in` of a warp.
    void choose(const std::vector<const GateDesc*>& g, const std::vector<int>& in, bool first) {
        int use[16] = {0};
        int pair[2] = {-1, -1};
        for (const GateDesc* x : g) {
            ++use[x->b0];
            if (x->op != 2) continue;
            ++use[x->b1];
            if (pair[0] < 0) {
                pair[0] = x->b0;
                pair[1] = x->b1;
            }
        }
        int next[16], n = 0;
        bool used[16] = {false};
        std::fill(next, next + 16, -1);
        std::vector<int> rest;
        if (f32) {
            // register slots: the first 2-qubit gate's bits, then the most used
            if (pair[0] >= 0) rest = {pair[1], pair[0]};
            std::vector<int> r;
            for (int b : in)
                if (b != pair[0] && b != pair[1]) r.push_back(b);
            std::stable_sort(r.begin(), r.end(), [&](int x, int y) { return use[x] > use[y]; });
            rest.insert(rest.end(), r.begin(), r.end());
        } else {
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
            for (int b : in)
                if (!used[b]) rest.push_back(b);
            std::stable_sort(rest.begin(), rest.end(), [&](int x, int y) { return use[x] > use[y]; });
        }
        for (int s = 0; s < NR; ++s) {
            next[s] = rest[size_t(n)];
            used[rest[size_t(n++)]] = true;
        }
        // the other lane slots: first bits whose shared-memory columns differ
        // from those of the lane slots before them (element bits of one class
        // modulo 3, in complex64 above bit 0, share a column)
        std::vector<int> lanes(rest.begin() + n, rest.end());
        auto cls = [&](int b) { return !f32 ? b % 3 : b == 0 ? 3 : (b - 1) % 3; };
        uint32_t cols = f32 ? 0u : (1u << cls(pair[0])) | (1u << cls(pair[1]));
        for (size_t x = 0; x < lanes.size(); ++x) {
            for (size_t y = x; y < lanes.size(); ++y)
                if (!((cols >> cls(lanes[y])) & 1u)) {
                    std::swap(lanes[x], lanes[y]);
                    break;
                }
            cols |= 1u << cls(lanes[x]);
            const int slot = NR + (f32 ? 0 : 2) + int(x);
            next[slot] = lanes[x];
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

    // Complex64: brings g's bits into register slots, each for the bit there
    // whose next use in the stretch (`when`) is the farthest.
    void to_regs(const GateDesc& g, const std::function<int(int)>& when) {
        int b[2] = {g.b0, g.op == 2 ? g.b1 : g.b0};
        for (int x = 0; x < g.op; ++x) {
            const int s = slot_of(b[x]);
            if (s < NR) continue;
            int victim = -1, far = -1;
            for (int r = 0; r < NR; ++r) {
                if (at[r] == b[0] || at[r] == b[1]) continue;
                const int w = when(at[r]);
                if (w > far) {
                    far = w;
                    victim = r;
                }
            }
            op(kRtSwap, s - NR, victim);
            std::swap(at[s], at[victim]);
        }
        if (g.op == 2 && ordered && slot_of(g.b1) > slot_of(g.b0)) {
            const int lo = slot_of(g.b0), hi = slot_of(g.b1);
            op(kRtTrade, lo, hi);
            std::swap(at[lo], at[hi]);
        }
    }

    // The moves that gate g (bits local to the tile) needs now.
    int moves(const GateDesc& g) const {
        if (f32) {
            int m = slot_of(g.b0) < NR ? 0 : 1;
            if (g.op == 2 && slot_of(g.b1) >= NR) ++m;
            return m;
        }
        if (g.op == 1) return slot_of(g.b0) < NR ? 0 : 3; // a shuffle of every register
        int m = 0;
        for (int b : {g.b0, g.b1}) {
            const int s = slot_of(b);
            m += s == NR || s == NR + 1 ? 0 : 1;
        }
        return m;
    }

    // Applies g with its controls on tile bits (local) and on others.
    void gate(const GateDesc& g, const std::vector<std::pair<int, int>>& local,
              const std::vector<std::pair<int, int>>& outside, const std::function<int(int)>& when) {
        RtOp o;
        std::memset(&o, 0, sizeof(o));
        if (f32) {
            to_regs(g, when);
            const int s0 = slot_of(g.b0), s1 = g.op == 2 ? slot_of(g.b1) : s0;
            o.type = g.op == 2 ? kRtG2 : kRtG1R;
            o.a = uint8_t(std::min(s0, s1));
            o.b = uint8_t(std::max(s0, s1));
        } else if (g.op == 2) {
            to_pair(g.b0, g.b1);
            o.type = kRtG2;
        } else {
            const int s = slot_of(g.b0);
            o.type = s < NR ? kRtG1R : kRtG1L;
            o.a = uint8_t(s < NR ? s : s - NR);
        }
        o.coef = uint32_t(f32 ? coef32.size() / 2 : coef.size());
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
        if (f32) { // row-major over the index bit a + 2 bit b
            const int D = g.op == 1 ? 2 : 4;
            const bool turn = g.op == 2 && o.a == slot_of(g.b0); // b0 is the low bit
            auto at4 = [&](int k) { return turn ? (k & 1) << 1 | k >> 1 : k; };
            for (int r = 0; r < D; ++r)
                for (int c = 0; c < D; ++c) {
                    const cd u = g.op == 1 ? g.A[r + 2 * c] : g.A[at4(r) + 4 * at4(c)];
                    coef32.push_back({float(u.real()), float(u.imag())});
                }
            return;
        }
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

size_t reg_program_bytes(const std::vector<GateDesc>& gates) {
    size_t b = 0; // every gate at most in a pass of its own
    for (const GateDesc& g : gates) b += kGateBytes[g.op] + 64 + kRtHeadBytes;
    return b;
}

void plan_reg_program(const std::vector<GateDesc>& gates, int nbits, int Tmax, RegProgram& P,
                      const std::function<void(const RegPass&)>& planned, bool ordered) {
    const bool f32 = P.prec == QGPU_C64;
    P.nbits = nbits;
    P.trades = f32 && ordered;
    P.passes.clear();
    P.single.clear();
    P.blob.clear();
    P.blob.reserve(reg_program_bytes(gates));
    int T, L, NR;
    reg_tile_shape(P.prec, nbits, Tmax, T, L, NR);
    const int nfree = T - L;
    const uint64_t low = (uint64_t(1) << L) - 1, every = (uint64_t(1) << std::max(nbits, T)) - 1;
    std::vector<Waiting> wait, pass, run;
    wait.reserve(std::min(gates.size(), kLookAhead));
    size_t next = 0; // the first gate that is not in `wait` yet
    auto refill = [&] {
        for (; next < gates.size() && wait.size() < kLookAhead; ++next) {
            const GateDesc& g = gates[next];
            Waiting w;
            w.t = uint64_t(1) << g.b0;
            if (g.op == 2) w.t |= uint64_t(1) << g.b1;
            w.a = w.t;
            for (const auto& c : g.ctrl) w.a |= uint64_t(1) << c.first;
            w.id = uint32_t(next);
            w.weight = uint32_t(g.op);
            wait.push_back(w);
        }
    };
    std::vector<GateDesc> loc; // the pass's gates on tile bits
    for (refill(); !wait.empty(); refill()) {
        const uint64_t S = choose_bits(wait, low, every, T);
        pass.clear();
        take(wait, S, (f32 ? kRt32BlobMax - kRtHeadBytes : kRtBlobMax) - 64, pass);
        if (pass.empty()) raise(QGPU_ERR_NOT_SUPPORTED, "qgpu_run_gates()", "tile too small");
        RegPass p;
        std::memset(&p, 0, sizeof(p));
        p.T = T;
        p.L = L;
        p.NR = NR;
        int nh = 0;
        for (int b = L; b < 64 && nh < nfree; ++b)
            if ((S >> b) & 1u) p.hi[nh++] = b;
        p.ntiles = nbits > T ? uint64_t(1) << (nbits - T) : 1;
        p.nvalid = nbits < T ? 1u << nbits : 1u << T;
        p.ngates = uint32_t(pass.size());
        p.single = -1;
        if (pass.size() == 1 && gates[pass[0].id].ctrl.empty()) {
            p.single = int(P.single.size());
            P.single.push_back(gates[pass[0].id]);
        }
        auto local = [&](int b) {
            return b < L ? b : L + int(std::find(p.hi, p.hi + nh, b) - p.hi);
        };
        // the gates on tile bits, numbered within the pass; controls outside
        // the tile stay where they are (and order nothing inside it: a gate
        // on such a bit is not in this pass)
        loc.resize(pass.size());
        for (size_t k = 0; k < pass.size(); ++k) {
            loc[k] = gates[pass[k].id];
            Waiting w;
            w.id = uint32_t(k);
            loc[k].b0 = local(loc[k].b0);
            w.t = uint64_t(1) << loc[k].b0;
            if (loc[k].op == 2) {
                loc[k].b1 = local(loc[k].b1);
                w.t |= uint64_t(1) << loc[k].b1;
            }
            w.a = w.t;
            for (const auto& c : loc[k].ctrl)
                if ((S >> c.first) & 1u) w.a |= uint64_t(1) << local(c.first);
            w.weight = pass[k].weight;
            pass[k] = w;
        }
        Builder B;
        B.f32 = f32;
        B.ordered = ordered;
        B.T = T;
        B.NR = NR;
        B.inwarp = NR + 5;
        bool first = true;
        while (!pass.empty()) {
            // a stretch of gates on the bits of one warp
            const uint64_t W = choose_bits(pass, 0, (uint64_t(1) << T) - 1, B.inwarp);
            run.clear();
            take(pass, W, ~size_t(0), run);
            std::vector<int> in;
            for (int b = 0; b < T; ++b)
                if ((W >> b) & 1u) in.push_back(b);
            std::vector<const GateDesc*> rg;
            for (const Waiting& w : run) rg.push_back(&loc[w.id]);
            B.choose(rg, in, first);
            first = false;
            // next the gate that needs the fewest moves among those whose
            // bits no earlier one of the stretch still waits for
            while (!run.empty()) {
                uint64_t seen = 0;
                size_t pick = 0;
                int least = 99;
                for (size_t k = 0; k < run.size() && least; ++k) {
                    if (!(run[k].a & seen)) {
                        const int m = B.moves(loc[run[k].id]);
                        if (m < least) {
                            least = m;
                            pick = k;
                        }
                    }
                    seen |= run[k].a;
                }
                const GateDesc& g = loc[run[pick].id];
                std::vector<std::pair<int, int>> inside, outside;
                for (auto& c : g.ctrl) {
                    if ((S >> c.first) & 1u) inside.push_back({local(c.first), c.second});
                    else outside.push_back(c);
                }
                const uint32_t id = run[pick].id;
                B.gate(g, inside, outside, [&](int bit) { // gates until the bit is used next
                    int n = 0;
                    for (const Waiting& w : run) {
                        if (w.id != id && ((w.t >> bit) & 1u)) return n;
                        ++n;
                    }
                    return 1000;
                });
                run.erase(run.begin() + ptrdiff_t(pick));
            }
        }
        B.table();
        p.nops = uint32_t(B.ops.size());
        p.nlay = uint32_t(B.lays.size());
        p.blob = uint32_t(P.blob.size());
        const size_t b_head = f32 ? kRtHeadBytes : 0;
        const size_t b_ops = (B.ops.size() * sizeof(RtOp) + 15) / 16 * 16;
        const size_t b_lay = B.lays.size() * sizeof(RtLayoutTab);
        const size_t b_coef = f32 ? B.coef32.size() * 8 : B.coef.size() * sizeof(cd);
        p.blob_bytes = uint32_t(b_head + b_ops + b_lay + b_coef);
        P.blob.resize(P.blob.size() + p.blob_bytes);
        unsigned char* d = P.blob.data() + p.blob;
        if (f32) {
            RtHead h;
            std::memset(&h, 0, sizeof(h));
            h.nops = p.nops;
            h.nlay = p.nlay;
            h.nvalid = p.nvalid;
            h.T = p.T;
            h.L = p.L;
            h.NR = p.NR;
            std::copy(p.hi, p.hi + 16, h.hi);
            std::memcpy(d, &h, sizeof(h));
            d += b_head;
        }
        std::memcpy(d, B.ops.data(), B.ops.size() * sizeof(RtOp));
        std::memcpy(d + b_ops, B.lays.data(), b_lay);
        if (f32) std::memcpy(d + b_ops + b_lay, B.coef32.data(), b_coef);
        else std::memcpy(d + b_ops + b_lay, B.coef.data(), b_coef);
        P.passes.push_back(p);
        if (planned) planned(p);
    }
}

} // namespace qgpu
