// CPU check of the register QFT passes (plan_qft_reg, k_qft_reg): a host model runs
// every planned pass as the kernel does -- tiles read in the first round's layout,
// each round on its register bits with the kernel's phase factors, the buffer
// written where it was read, the last round's layout written out -- and must give
// the transform's definition within 1e-11 (10 to 17 steps in 64 bits, errors of a
// few ulp each), reading and writing inside the state, every element once, with
// each round's threads and registers covering the tile once and no bank conflicts
// in the rounds between the first and the last. Whole and partial transforms,
// ordered and scattered targets, both precisions' tiles, both directions, with and
// without the reversal. Whole transforms of 24 to 28 qubits take three passes, of 30 four (no three groups of ten targets).
// Built and run by tests/test_qft_reg.py.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

#include "kernels.hpp"

using namespace qgpu;
using cdd = std::complex<double>;

static int fails = 0;
#define EXPECT(c)                                                                     \
    do {                                                                              \
        if (!(c)) {                                                                   \
            if (fails < 20) std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #c); \
            ++fails;                                                                  \
        }                                                                             \
    } while (0)

static cdd turn(double x) { return cdd(std::cos(M_PI * x), std::sin(M_PI * x)); }

static uint32_t swz(int bits, uint32_t e) {
    return bits == 12 ? e ^ ((e >> 3) & 7u) ^ ((e >> 6) & 7u) ^ ((e >> 9) & 7u)
                   : e ^ ((e >> 4) & 15u) ^ ((e >> 8) & 15u) ^ ((e >> 12) & 15u);
}

static void check_layouts(const QftRegPlan& p) {
    const int NR = p.bits - kQftRegThrBits;
    for (int r = 0; r < p.nround; ++r) {
        const QftRegRound& rd = p.rd[r];
        std::vector<int> seen(size_t(p.bits), 0);
        for (int i = 0; i < NR; ++i) seen[rd.reg[i]]++;
        for (int i = 0; i < kQftRegThrBits; ++i) seen[rd.thr[i]]++;
        for (int x : seen) EXPECT(x == 1);
        for (int i = 0; i < rd.g; ++i) EXPECT(rd.reg[i] == rd.lo + i);
        if (rd.g) { // no phase reaches a register bit but those of the round
            EXPECT(rd.lo >= p.nr && rd.g <= NR);
            for (int i = 0; i < NR; ++i) EXPECT(rd.reg[i] >= rd.lo);
        }
        if (r > 0 && r + 1 < p.nround) {
            const uint32_t lanes = p.bits == 12 ? 8 : 16;
            std::vector<int> hit(lanes, 0);
            for (uint32_t l = 0; l < lanes; ++l) {
                uint32_t e = 0;
                for (int i = 0; i < kQftRegThrBits; ++i) e |= ((l >> i) & 1u) << rd.thr[i];
                hit[swz(p.bits, e) % lanes]++;
            }
            for (int x : hit) EXPECT(x == 1);
        }
    }
    uint64_t rmax = 0, wmax = 0, tiles = 1;
    for (int q = 0; q < p.nod; ++q) {
        rmax += (p.odim[q] - 1) * p.ors[q];
        wmax += (p.odim[q] - 1) * p.ows[q];
        EXPECT(tiles == uint64_t(1) << p.oshift[q]);
        tiles *= p.odim[q];
    }
    EXPECT(tiles == p.ntiles);
    for (int b = 0; b < p.bits; ++b) rmax += p.trs[b], wmax += p.tws[b];
    EXPECT(rmax + 1 == p.ntiles << p.bits && wmax + 1 == p.ntiles << p.bits);
    // dynamic shared memory of two CTAs per SM
    EXPECT((65536 + size_t((1 << (p.M - 1)) + (p.M << p.nz) + 4 * p.M) * 16 + size_t(p.nround) * 512 + 4224) * 2 <= 226 * 1024);
}

static void run_pass(const QftRegPlan& p, const std::vector<cdd>& in,
                     std::vector<cdd>& out) {
    const int NR = p.bits - kQftRegThrBits;
    const double s = p.inverse ? -1 : 1;
    std::vector<int> wrote(out.size(), 0);
    std::vector<cdd> v(size_t(1) << p.bits), buf(size_t(1) << p.bits);
    for (uint64_t t = 0; t < p.ntiles; ++t) {
        uint64_t rb = 0, wb = 0, z = 0;
        for (int q = 0; q < p.nod; ++q) {
            const uint64_t dg = (t >> p.oshift[q]) & (p.odim[q] - 1);
            rb += dg * p.ors[q], wb += dg * p.ows[q], z += dg * p.ozw[q];
        }
        for (int r = 0; r < p.nround; ++r) {
            const QftRegRound& rd = p.rd[r];
            for (uint32_t tid = 0; tid < (1u << kQftRegThrBits); ++tid) {
                uint32_t e = 0;
                for (int i = 0; i < kQftRegThrBits; ++i) e |= ((tid >> i) & 1u) << rd.thr[i];
                cdd x[32];
                uint32_t pos[32];
                for (int m = 0; m < (1 << NR); ++m) {
                    pos[m] = e;
                    for (int i = 0; i < NR; ++i) pos[m] |= uint32_t((m >> i) & 1) << rd.reg[i];
                    uint64_t a = rb;
                    for (int b = 0; b < p.bits; ++b) a += ((pos[m] >> b) & 1u) * p.trs[b];
                    if (r == 0) EXPECT(a < in.size());
                    x[m] = r == 0 ? in[a] : buf[swz(p.bits, pos[m])];
                }
                for (int u = 0; u < rd.g; ++u) {
                    const int rel = p.inverse ? u : rd.g - 1 - u, j = p.nr + p.M - 1 - rd.lo - rel;
                    const uint32_t L = (e >> p.nr) & ((1u << (rd.lo - p.nr)) - 1);
                    uint64_t zz = z;
                    for (int q = 0; q < p.nz; ++q) zz += uint64_t((e >> q) & 1u) * p.tzw[q];
                    const cdd b = turn(s * (std::ldexp(double(L), 1 + j - p.M) +
                                            std::ldexp(double(zz), 1 - (p.k - p.a - j))));
                    for (int m = 0; m < (1 << NR); ++m) {
                        if ((m >> rel) & 1) continue;
                        const int lb = m & ((1 << rel) - 1), m1 = m | (1 << rel);
                        const cdd ph = b * turn(s * lb / double(1 << rel));
                        const cdd y = p.inverse ? x[m1] * ph : x[m1], a = x[m];
                        x[m] = a + y;
                        x[m1] = p.inverse ? a - y : (a - y) * ph;
                    }
                }
                for (int m = 0; m < (1 << NR); ++m) {
                    if (r + 1 < p.nround) {
                        v[swz(p.bits, pos[m])] = x[m];
                        continue;
                    }
                    uint64_t a = wb;
                    for (int b = 0; b < p.bits; ++b) a += ((pos[m] >> b) & 1u) * p.tws[b];
                    EXPECT(a < out.size());
                    out[a] = x[m] * p.scale;
                    wrote[a]++;
                }
            }
            buf = v;
        }
    }
    for (int w : wrote) EXPECT(w == 1);
}

// the definition: on the targets' value, sum over y of exp(s 2 pi i x y / 2^k); with
// the reversal the result as it is, without it at the reversed digits
static std::vector<cdd> exact(const std::vector<cdd>& in, int n, const std::vector<uint64_t>& tg, bool inv,
                              bool rev) {
    // step by step on single digits, as the header of kernels_qft.cu states them
    std::vector<cdd> a = in;
    const size_t k = tg.size();
    auto bit = [&](uint64_t q) { return n - 1 - int(q); };
    auto swap_all = [&] {
        if (!rev) return;
        for (size_t i = 0; i < k / 2; ++i) {
            const uint64_t x = uint64_t(1) << bit(tg[i]), y = uint64_t(1) << bit(tg[k - 1 - i]);
            for (uint64_t e = 0; e < a.size(); ++e)
                if ((e & x) && !(e & y)) std::swap(a[e], a[(e ^ x) | y]);
        }
    };
    if (inv) swap_all();
    for (size_t u = 0; u < k; ++u) {
        const size_t i = inv ? k - 1 - u : u;
        const uint64_t b = uint64_t(1) << bit(tg[i]);
        for (uint64_t e = 0; e < a.size(); ++e) {
            if (e & b) continue;
            double Y = 0;
            for (size_t l = i + 1; l < k; ++l) Y = 2 * Y + double((e >> bit(tg[l])) & 1u);
            const cdd ph = turn((inv ? -1.0 : 1.0) * 2 * Y / std::ldexp(1.0, int(k - i)));
            const cdd x = a[e], y = inv ? a[e | b] * ph : a[e | b];
            a[e] = (x + y) * M_SQRT1_2;
            a[e | b] = (x - y) * M_SQRT1_2 * (inv ? cdd(1) : ph);
        }
    }
    if (!inv) swap_all();
    return a;
}

int main() {
    std::mt19937 gen(7);
    std::normal_distribution<double> g;
    int ran = 0;
    for (qgpu_prec prec : {QGPU_C128, QGPU_C64})
        for (int n : {13, 14, 17})
            for (int k : {9, 10, 11, 12, 13, 17})
                for (int scattered = 0; scattered < 2; ++scattered)
                    for (int inv = 0; inv < 2; ++inv)
                        for (int rev = 0; rev < 2; ++rev) {
                            if (k > n) continue;
                            std::vector<uint64_t> all;
                            for (int i = 0; i < n; ++i) all.push_back(uint64_t(i));
                            if (scattered) std::shuffle(all.begin(), all.end(), gen);
                            const std::vector<uint64_t> t(all.begin(), all.begin() + k);
                            QftRegSchedule S;
                            if (!plan_qft_reg(prec, uint64_t(1) << n, t, inv != 0, rev != 0, S)) continue;
                            ++ran;
                            std::vector<cdd> a(size_t(1) << n);
                            for (cdd& x : a) x = cdd(g(gen), g(gen));
                            const std::vector<cdd> want = exact(a, n, t, inv != 0, rev != 0);
                            for (size_t i = 0; i < S.plans.size(); ++i) {
                                const QftRegPlan& p = S.plans[i];
                                check_layouts(p);
                                std::vector<cdd> b(a.size());
                                run_pass(p, a, b);
                                if (!S.fold[i])
                                    for (int q = 0; q < p.bits; ++q) EXPECT(p.trs[q] == p.tws[q]);
                                a.swap(b);
                            }
                            double err = 0, big = 0;
                            for (size_t i = 0; i < a.size(); ++i) {
                                err = std::max(err, std::abs(a[i] - want[i]));
                                big = std::max(big, std::abs(want[i]));
                            }
                            EXPECT(err <= 1e-11 * big);
                        }
    EXPECT(ran >= 100);
    for (qgpu_prec prec : {QGPU_C128, QGPU_C64})
        for (int n = 24; n <= 30; ++n)
            for (int inv = 0; inv < 2; ++inv)
                for (int rev = 0; rev < 2; ++rev) {
                    std::vector<uint64_t> t;
                    for (int i = 0; i < n; ++i) t.push_back(uint64_t(i));
                    QftRegSchedule S;
                    EXPECT(plan_qft_reg(prec, uint64_t(1) << n, t, inv != 0, rev != 0, S));
                    EXPECT(S.plans.size() == (n < 29 || (n == 29 && prec == QGPU_C64) ? 3u : 4u));
                    for (const QftRegPlan& p : S.plans) check_layouts(p);
                }
    std::printf("%d transforms\n", ran);
    std::printf(fails ? "qft reg FAILED (%d)\n" : "qft reg ok\n", fails);
    return fails ? 1 : 0;
}
