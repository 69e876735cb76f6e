// CPU check of the register tile passes (qgpu::plan_reg_program): a host model
// of k_reg_tile and k_reg_tile32 -- the tile spread over
// registers, lanes and warps, the shuffles, the layout changes through shared
// memory and the matrix fragments of the 2-qubit gates -- runs the planned
// programs of random 1- and 2-qubit gates with 0-3 controls on kets of 1-15
// qubits and must give the gates applied one by one (in circuit order) within
// 1e-13 (relative, max-norm: 60 gates of unit-norm rows, each at most a few
// ulp) in complex128, 3e-5 with complex64 coefficients. Every pass must touch each amplitude once, keep its shared memory
// inside the kernel's limit and hold only positions inside its tile. Built and
// run by tests/test_reg_tiles.py.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "reg_tiles.hpp"

using namespace qgpu;
using C = std::complex<double>;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            if (fails < 20) std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c);   \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

static void apply_direct(std::vector<C>& psi, const GateDesc& g) {
    const uint64_t N = psi.size(), s0 = uint64_t(1) << g.b0, s1 = g.op == 2 ? uint64_t(1) << g.b1 : 0;
    for (uint64_t i = 0; i < N; ++i) {
        if ((i & s0) || (i & s1)) continue;
        bool ok = true;
        for (auto& c : g.ctrl) ok = ok && int((i >> c.first) & 1) == c.second;
        if (!ok) continue;
        const int D = g.op == 1 ? 2 : 4;
        const uint64_t at[4] = {i, g.op == 1 ? i + s0 : i + s1, i + s0, i + s0 + s1};
        C v[4], r[4];
        for (int k = 0; k < D; ++k) v[k] = psi[at[k]];
        for (int k = 0; k < D; ++k) {
            r[k] = 0;
            for (int c = 0; c < D; ++c) r[k] += g.A[k + D * c] * v[c];
        }
        for (int k = 0; k < D; ++k) psi[at[k]] = r[k];
    }
}

// host model of k_reg_tile (f32: of k_reg_tile32, in double arithmetic) on one
// pass
static void run_pass(std::vector<C>& psi, const RegPass& p, const unsigned char* blob,
                     std::vector<int>& visits, bool f32) {
    const unsigned char* const end = blob + p.blob_bytes;
    if (f32) {
        const auto* h = reinterpret_cast<const RtHead*>(blob);
        EXPECT(h->nops == p.nops && h->nlay == p.nlay && h->nvalid == p.nvalid && h->T == p.T &&
               h->L == p.L && h->NR == p.NR && std::equal(p.hi, p.hi + 16, h->hi));
        blob += kRtHeadBytes;
    }
    auto swz = [&](uint32_t e) { return f32 ? rt_swz32(e) : rt_swz(e); };
    const int T = p.T, NR = p.NR, R = 1 << NR, W = 1 << (T - NR - 5), nth = 32 * W, nhi = T - p.L;
    const auto* ops = reinterpret_cast<const RtOp*>(blob);
    const auto* lays = reinterpret_cast<const RtLayoutTab*>(blob + (p.nops * sizeof(RtOp) + 15) / 16 * 16);
    // entry k of the coefficients from 16-byte unit u on
    const auto* tables = reinterpret_cast<const unsigned char*>(lays + p.nlay);
    auto entry = [&](uint32_t u, int k) -> C {
        if (f32) {
            const auto* x = reinterpret_cast<const std::complex<float>*>(tables) + 2 * u + k;
            EXPECT(reinterpret_cast<const unsigned char*>(x + 1) <= end);
            return C(x->real(), x->imag());
        }
        const C* x = reinterpret_cast<const C*>(tables) + u + k;
        EXPECT(reinterpret_cast<const unsigned char*>(x + 1) <= end);
        return *x;
    };
    EXPECT((size_t(f32 ? 8 : 16) << T) + ((size_t(8) << nhi) + 15) / 16 * 16 + p.blob_bytes <=
           (f32 ? kRt32SmemMax : kRtSmemMax));
    const uint32_t nel = 1u << T;
    std::vector<C> tile(nel), v(size_t(nth) * R), w;
    auto at = [&](int lay, int th, int j) {
        uint32_t b = 0;
        for (int k = 0; k < NR; ++k)
            if (j >> k & 1) b ^= lays[lay].img[k];
        for (int k = 0; k < T - NR; ++k)
            if (th >> k & 1) b ^= lays[lay].img[NR + k];
        EXPECT(b < nel);
        return b % nel;
    };
    auto put = [&](int lay) { // every position once
        std::vector<int> seen(nel, 0);
        for (int th = 0; th < nth; ++th)
            for (int j = 0; j < R; ++j) {
                tile[at(lay, th, j)] = v[size_t(th) * R + j];
                ++seen[at(lay, th, j)];
            }
        for (uint32_t e = 0; e < nel; ++e) EXPECT(seen[e] == 1);
    };
    auto get = [&](int lay) {
        for (int th = 0; th < nth; ++th)
            for (int j = 0; j < R; ++j) v[size_t(th) * R + j] = tile[at(lay, th, j)];
    };
    for (uint64_t t = 0; t < p.ntiles; ++t) {
        uint64_t base = t << p.L;
        for (int i = 0; i < nhi; ++i) {
            const uint64_t low = (uint64_t(1) << p.hi[i]) - 1;
            base = ((base & ~low) << 1) | (base & low);
        }
        auto addr = [&](uint32_t e) {
            uint64_t a = base + (e & ((1u << p.L) - 1));
            for (int i = 0; i < nhi; ++i)
                if ((e >> (p.L + i)) & 1u) a += uint64_t(1) << p.hi[i];
            return a;
        };
        for (uint32_t e = 0; e < nel; ++e) {
            tile[swz(e)] = 0;
            if (e >= p.nvalid) continue;
            EXPECT(addr(e) < psi.size());
            tile[swz(e)] = psi[addr(e)];
            ++visits[addr(e)];
        }
        get(0);
        for (uint32_t o = 0; o < p.nops; ++o) {
            const RtOp& op = ops[o];
            if (op.type <= kRtG1L) {
                w = v;
                for (int th = 0; th < nth; ++th) {
                    const int lane = th & 31, warp = th >> 5;
                    for (int j = 0; j < R; ++j) {
                        C r = 0;
                        if (op.type == kRtG2 && f32) {
                            EXPECT(op.a < op.b && op.b < NR);
                            const int k = (j >> op.a & 1) | (j >> op.b & 1) << 1;
                            for (int c = 0; c < 4; ++c) {
                                const int jc = (j & ~(1 << op.a) & ~(1 << op.b)) | (c & 1) << op.a | (c >> 1) << op.b;
                                r += entry(op.coef, 4 * k + c) * w[size_t(th) * R + jc];
                            }
                        } else if (op.type == kRtG2) {
                            // row lane >> 2 of the 8 x 4 operand, column pair
                            // 2 (lane & 3) of the product
                            double d[2] = {0, 0};
                            for (int x = 0; x < 2; ++x)
                                for (int k = 0; k < 4; ++k) {
                                    const C a = w[size_t((th & ~3) + k) * R + j];
                                    const C b = entry(op.coef, 4 * (2 * (lane & 3) + x) + k);
                                    d[x] += a.real() * b.real() + a.imag() * b.imag();
                                }
                            r = C(d[0], d[1]);
                        } else if (op.type == kRtG1R) {
                            EXPECT(op.a < NR);
                            const int s = j >> op.a & 1, j0 = j & ~(1 << op.a);
                            r = entry(op.coef, 2 * s) * w[size_t(th) * R + j0] +
                                entry(op.coef, 2 * s + 1) * w[size_t(th) * R + (j0 | 1 << op.a)];
                        } else {
                            EXPECT(op.a < 5 && !f32);
                            const int s = lane >> op.a & 1;
                            r = entry(op.coef, 3 * s) * w[size_t(th) * R + j] +
                                entry(op.coef, 1 + s) * w[size_t(th ^ (1 << op.a)) * R + j];
                        }
                        const bool ok = !op.ctrl || ((base & op.gmask) == op.gval && (warp & op.wmask) == op.wval &&
                                                     (lane & op.lmask) == op.lval && (j & op.rmask) == op.rval);
                        if (ok) v[size_t(th) * R + j] = r;
                    }
                }
            } else if (op.type == kRtSwap) {
                EXPECT(op.a < 5 && op.b < NR);
                w = v;
                for (int th = 0; th < nth; ++th)
                    for (int j = 0; j < R; ++j) {
                        const int x = th >> op.a & 1, y = j >> op.b & 1;
                        const int th2 = (th & ~(1 << op.a)) | y << op.a, j2 = (j & ~(1 << op.b)) | x << op.b;
                        v[size_t(th) * R + j] = w[size_t(th2) * R + j2];
                    }
            } else if (op.type == kRtTrade) {
                EXPECT(f32 && op.a < op.b && op.b < NR);
                w = v;
                for (int th = 0; th < nth; ++th)
                    for (int j = 0; j < R; ++j) {
                        const int x = j >> op.a & 1, y = j >> op.b & 1;
                        const int j2 = (j & ~(1 << op.a) & ~(1 << op.b)) | y << op.a | x << op.b;
                        v[size_t(th) * R + j] = w[size_t(th) * R + j2];
                    }
            } else if (op.type == kRtPerm) {
                EXPECT(!f32);
                w = v;
                for (int th = 0; th < nth; ++th) {
                    int src = th & ~31;
                    for (int i = 0; i < 5; ++i) src |= (th >> i & 1) << (op.coef >> (3 * i) & 7);
                    for (int j = 0; j < R; ++j) v[size_t(th) * R + j] = w[size_t(src) * R + j];
                }
            } else {
                EXPECT(op.type == kRtLayout && op.coef + 1 < p.nlay);
                put(int(op.coef));
                get(int(op.coef) + 1);
            }
        }
        put(int(p.nlay) - 1);
        for (uint32_t e = 0; e < nel; ++e)
            if (e < p.nvalid) psi[addr(e)] = tile[swz(e)];
    }
}

int main() {
    std::mt19937_64 rng(11);
    std::normal_distribution<double> nd;
    int cases = 0;
    for (int nbits = 1; nbits <= 15; ++nbits)
        for (int Tmax : {5, 8, 9, 11, 12}) {
            std::vector<GateDesc> gates;
            for (int k = 0; k < 60; ++k) {
                std::vector<int> perm(nbits);
                for (int i = 0; i < nbits; ++i) perm[i] = i;
                std::shuffle(perm.begin(), perm.end(), rng);
                GateDesc g;
                g.op = nbits >= 2 && rng() % 2 ? 2 : 1;
                g.b0 = perm[0];
                if (g.op == 2) g.b1 = perm[1];
                const int nc = rng() % 3 ? 0 : int(rng() % 4);
                for (int i = 0; i < nc && g.op + i < nbits; ++i) g.ctrl.push_back({perm[g.op + i], int(rng() % 2)});
                const int D = 1 << g.op;
                for (int r = 0; r < D; ++r) { // rows of unit norm
                    double s = 0;
                    for (int c = 0; c < D; ++c) s += std::norm(g.A[r + D * c] = C(nd(rng), nd(rng)));
                    for (int c = 0; c < D; ++c) g.A[r + D * c] /= std::sqrt(s);
                }
                gates.push_back(g);
            }
            std::vector<C> psi(size_t(1) << nbits);
            for (auto& x : psi) x = C(nd(rng), nd(rng));
            std::vector<C> ref = psi;
            for (const auto& g : gates) apply_direct(ref, g);
            for (int form = 0; form < 3; ++form) { // complex128; complex64, also ordered
                RegProgram P;
                P.prec = form ? QGPU_C64 : QGPU_C128;
                plan_reg_program(gates, nbits, Tmax, P, nullptr, form == 2);
                std::vector<C> got = psi;
                uint32_t covered = 0;
                for (const RegPass& p : P.passes) {
                    EXPECT(p.blob % 16 == 0 && p.blob + p.blob_bytes <= P.blob.size());
                    EXPECT(p.single < 0 || (p.ngates == 1 && P.single[size_t(p.single)].ctrl.empty()));
                    covered += p.ngates;
                    std::vector<int> visits(psi.size(), 0);
                    run_pass(got, p, P.blob.data() + p.blob, visits, form > 0);
                    for (int x : visits) EXPECT(x == 1);
                }
                EXPECT(covered == gates.size());
                double top = 0, err = 0;
                for (size_t i = 0; i < ref.size(); ++i) {
                    top = std::max(top, std::abs(ref[i]));
                    err = std::max(err, std::abs(got[i] - ref[i]));
                }
                EXPECT(err <= (form ? 3e-5 : 1e-13) * top);
                ++cases;
            }
        }
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("reg tiles ok: %d cases\n", cases);
    return 0;
}
