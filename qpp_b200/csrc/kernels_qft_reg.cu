// kernels_qft_reg.cu -- qubit Fourier transform passes of up to 10 steps (sm_100a).
//
// The steps and phases are those of kernels_qft.cu; here a tile is 64 KB, held in
// registers (16 complex128 or 32 complex64 amplitudes to each of 256 threads), so
// that a pass takes 9 or 10 targets where the tiles in shared memory take 8: 28
// qubits in three passes over the state instead of four. A round runs the steps on
// its register bits; between rounds the amplitudes change owner through a 64 KB
// shared-memory buffer (written where they were read, one barrier). The first round
// reads global memory straight into registers and the last one writes it, lanes over
// the lowest address bits. Two CTAs per SM: one's loads run under the other's steps.
//
// Phase of a step whose bit is register bit `rel`: the digits below it are `rel`
// register bits (value lb), thread bits, later targets in the tile's run digits and
// later targets outside the tile. The last three are one factor per thread and step
// (W T[j][c] B[j]); the first is a constant, exp(2 pi i lb / 2^(rel + 1)).
//
// Also below the L2 size: fewer passes and 4 instead of 3 steps a round; 20 qubits
// complex128 62 -> 34 us, 12 qubits 28 -> 17 us (one tile, two passes), most of it
// launches.
//
// Bound by memory above it: 28 qubits complex128 take 2.00 + 1.86 + 2.49 ms (9, 9 and 10
// targets; the copy rate gives 1.31 a pass, these access patterns without the steps
// 1.76, 1.52 and 2.42: the last one writes runs of 64 bytes, as its ten group bits
// leave the tile two others). 8-target passes in shared memory took four passes, 7.8 to
// 8.2 ms. What the L1 has left beside the shared memory holds the accesses in
// flight: 92 KB at two CTAs of 80 KB, with 60 KB the first pass took 2.28 ms and with 28
// KB 2.74; hence one buffer, small tables, nothing spilled to local memory. Tried and
// slower: 512 threads of 8 amplitudes (2.5 ms), a third buffer for the next tile
// filled by cp.async under one 512-thread CTA (3.3 ms), a factor per step and
// thread in place of W and T (2.65 ms, 107 KB).
#include <algorithm>

#include "kernels.hpp"

namespace qgpu {

namespace {

constexpr int kThr = 256;

template <typename R>
struct RegShape {
    static constexpr int NR = sizeof(R) == 8 ? 4 : 5; // log2 of a thread's amplitudes
    static constexpr int EB = 8 + NR;
};

__device__ __forceinline__ double2 ld_stream(const double2* a) {
    double2 v;
    asm volatile("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_stream(const float2* a) {
    float2 v;
    asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(a) : "memory");
    return v;
}

// buffer position of tile index e: the lanes that share a 128-byte wavefront (8 of
// 16 bytes, 16 of 8) hit distinct banks when their index bits have distinct
// residues modulo 3 (4)
template <typename R>
__device__ __forceinline__ uint32_t qft_reg_swz(uint32_t e) {
    return sizeof(R) == 8 ? e ^ ((e >> 3) & 7u) ^ ((e >> 6) & 7u) ^ ((e >> 9) & 7u)
                          : e ^ ((e >> 4) & 15u) ^ ((e >> 8) & 15u) ^ ((e >> 12) & 15u);
}

// cos(2 pi q / 32), q = 0..8
__host__ __device__ constexpr double cos32(int q) {
    constexpr double c[9] = {1.0,
                             0.98078528040323044913,
                             0.92387953251128675613,
                             0.83146961230254523708,
                             0.70710678118654752440,
                             0.55557023301960222474,
                             0.38268343236508977173,
                             0.19509032201612826785,
                             0.0};
    return c[q];
}

// a * exp(+-2 pi i q / 32), 0 <= q < 16, q a constant after unrolling
template <typename R, bool INV, typename C>
__device__ __forceinline__ C mul_root(C a, int q) {
    const R s = INV ? R(-1) : R(1);
    if (q == 0) return a;
    if (q == 8) return C{-s * a.y, s * a.x};
    const R c = q <= 8 ? R(cos32(q <= 8 ? q : 0)) : R(-cos32(q > 8 ? 16 - q : 0));
    const R n = s * R(cos32(q <= 8 ? 8 - q : q - 8)); // the sine, >= 0 for q < 16
    return C{a.x * c - a.y * n, a.x * n + a.y * c};
}

// G steps on the low G register bits. b[rel]: the thread's factor of the step on
// register bit rel.
template <typename R, bool INV, int G>
__device__ __forceinline__ void reg_steps(Cplx<R>* v, const double2* b) {
    using C = Cplx<R>;
    constexpr int NM = 1 << RegShape<R>::NR;
#pragma unroll
    for (int u = 0; u < G; ++u) {
        const int rel = INV ? u : G - 1 - u;
#pragma unroll
        for (int lb = 0; lb < (1 << (G - 1)); ++lb) {
            if (lb >= (1 << rel)) break;
            const double2 w = mul_root<double, INV>(b[rel], lb << (4 - rel));
            const C ph{R(w.x), R(w.y)};
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                if (((m >> rel) & 1) || (m & ((1 << rel) - 1)) != lb) continue;
                const int m1 = m | (1 << rel);
                const C x = v[m];
                if (!INV) {
                    const C y = v[m1];
                    v[m] = C{x.x + y.x, x.y + y.y};
                    v[m1] = cmul(C{x.x - y.x, x.y - y.y}, ph);
                } else {
                    const C y = cmul(v[m1], ph);
                    v[m] = C{x.x + y.x, x.y + y.y};
                    v[m1] = C{x.x - y.x, x.y - y.y};
                }
            }
        }
    }
}

} // namespace

template <typename R, bool INV, typename OFF>
__global__ void __launch_bounds__(kThr, 2)
    k_qft_reg(const Cplx<R>* in, Cplx<R>* out, const __grid_constant__ QftRegPlan p) {
    using C = Cplx<R>;
    constexpr int NR = RegShape<R>::NR, EB = RegShape<R>::EB, NM = 1 << NR;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* const buf = reinterpret_cast<C*>(smem_raw); // [2^EB]
    // the factors in 64 bits in both precisions: a complex64 step rounds its phase once
    // (error of 28 qubits against 64 bits 2.1e-7; 2.9e-7 with 32-bit factors, at 3.0
    // instead of 3.2 ms; four passes in shared memory 2.5e-7)
    double2* const W = reinterpret_cast<double2*>(buf + (1 << EB)); // [2^(M-1)]: exp(+-2 pi i e / 2^M)
    double2* const T = W + (1 << (p.M - 1));            // [M][2^nz]
    double2* const Bs = T + (p.M << p.nz);              // [4][M], by tile
    uint16_t* const eth = reinterpret_cast<uint16_t*>(Bs + 4 * p.M); // [nround][256]
    const int tid = threadIdx.x, M = p.M;
    const bool last_group = p.a + M == p.k; // no later targets: T = B = 1
    for (int i = tid; i < (1 << (M - 1)); i += kThr) {
        double sn, cs;
        sincospi(ldexp(double(i), 1 - M), &sn, &cs);
        W[i] = double2{cs, INV ? -sn : sn};
    }
    for (int i = tid; i < (M << p.nz); i += kThr) {
        const int j = i >> p.nz;
        uint64_t zz = 0;
        for (int q = 0; q < p.nz; ++q) zz += uint64_t((i >> q) & 1) * p.tzw[q];
        double sn, cs;
        sincospi(ldexp(double(zz), 1 - (p.k - p.a - j)), &sn, &cs);
        T[i] = double2{cs, INV ? -sn : sn};
    }
    for (int r = 0; r < p.nround; ++r) {
        uint32_t e = 0;
        for (int i = 0; i < kQftRegThrBits; ++i) e |= ((uint32_t(tid) >> i) & 1u) << p.rd[r].thr[i];
        eth[r * kThr + tid] = uint16_t(e);
    }
    auto tile_base = [&](uint64_t t, OFF& rb, OFF& wb, uint64_t& z) {
        rb = wb = 0;
        z = 0;
        for (int q = 0; q < p.nod; ++q) {
            const uint64_t dg = (t >> p.oshift[q]) & (p.odim[q] - 1);
            rb += OFF(dg * p.ors[q]);
            wb += OFF(dg * p.ows[q]);
            z += dg * p.ozw[q];
        }
    };
    auto set_b = [&](uint64_t z, double2* b) {
        if (tid < M) {
            double sn, cs;
            sincospi(ldexp(double(z), 1 - (p.k - p.a - tid)), &sn, &cs);
            b[tid] = double2{cs, INV ? -sn : sn};
        }
    };
    // the thread's offsets and the register bits' strides at both ends: in shared
    // memory, since kept in registers they would spill
    OFF* const offs = reinterpret_cast<OFF*>(eth + p.nround * kThr); // [2][256], [2][NR]
    {
        const QftRegRound& first = p.rd[0];
        const QftRegRound& last = p.rd[p.nround - 1];
        OFF oR = 0, oW = 0;
        for (int i = 0; i < kQftRegThrBits; ++i) {
            if ((tid >> i) & 1) {
                oR += OFF(p.trs[first.thr[i]]);
                oW += OFF(p.tws[last.thr[i]]);
            }
        }
        offs[tid] = oR;
        offs[kThr + tid] = oW;
        if (tid < NR) {
            offs[2 * kThr + tid] = OFF(p.trs[first.reg[tid]]);
            offs[2 * kThr + NR + tid] = OFF(p.tws[last.reg[tid]]);
        }
    }
    auto at = [&](const OFF* s, int m) {
        OFF o = 0;
#pragma unroll
        for (int i = 0; i < NR; ++i)
            if ((m >> i) & 1) o += s[i];
        return o;
    };

    uint64_t t = blockIdx.x;
    if (t >= p.ntiles) return;
    OFF rb, wb;
    uint64_t z;
    tile_base(t, rb, wb, z);
    set_b(z, Bs);
    __syncthreads();
    const R sc = R(p.scale);
    for (int it = 0; t < p.ntiles; t += gridDim.x, ++it) {
        const double2* const B = Bs + (it & 3) * M;
        C v[NM];
        {
            OFF st[NR];
#pragma unroll
            for (int i = 0; i < NR; ++i) st[i] = offs[2 * kThr + i];
            const C* const src = in + rb + offs[tid];
#pragma unroll
            for (int m = 0; m < NM; ++m) v[m] = ld_stream(src + at(st, m));
        }
        const uint64_t tn = t + gridDim.x;
        OFF wbn = 0;
        if (tn < p.ntiles) { // the next slot's last readers, of tile it - 3, are past a barrier of it - 1
            uint64_t zn;
            tile_base(tn, rb, wbn, zn);
            set_b(zn, Bs + ((it + 1) & 3) * M);
        }
        for (int r = 0;; ++r) {
            const QftRegRound& rd = p.rd[r];
            const uint32_t e = eth[r * kThr + tid], s0 = qft_reg_swz<R>(e);
            auto pos = [&](int m) {
                uint32_t s = s0;
#pragma unroll
                for (int i = 0; i < NR; ++i)
                    if ((m >> i) & 1) s ^= qft_reg_swz<R>(1u << rd.reg[i]);
                return s;
            };
            if (r > 0) {
#pragma unroll
                for (int m = 0; m < NM; ++m) v[m] = buf[pos(m)];
            }
            if (rd.g) {
                const int jlow = p.nr + M - 1 - rd.lo;
                const uint32_t L = (e >> p.nr) & ((1u << (rd.lo - p.nr)) - 1), c = e & ((1u << p.nz) - 1);
                double2 b[NR];
#pragma unroll
                for (int rel = 0; rel < NR; ++rel) {
                    if (rel >= rd.g) continue;
                    const int j = jlow - rel;
                    b[rel] = W[L << j];
                    if (!last_group) b[rel] = cmul(b[rel], cmul(B[j], T[(j << p.nz) + c]));
                }
                switch (rd.g) {
                    case 1: reg_steps<R, INV, 1>(v, b); break;
                    case 2: reg_steps<R, INV, 2>(v, b); break;
                    case 3: reg_steps<R, INV, 3>(v, b); break;
                    case 4: reg_steps<R, INV, 4>(v, b); break;
                    case 5:
                        if constexpr (NR == 5) reg_steps<R, INV, 5>(v, b);
                        break;
                    default: break;
                }
            }
            if (r + 1 == p.nround) break;
            // the first write waits until the previous tile's last round has read
            if (r == 0 && it > 0) __syncthreads();
#pragma unroll
            for (int m = 0; m < NM; ++m) buf[pos(m)] = v[m];
            __syncthreads();
        }
        OFF st[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) st[i] = offs[2 * kThr + NR + i];
        C* const dst = out + wb + offs[kThr + tid];
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            C x = v[m];
            x.x *= sc;
            x.y *= sc;
            dst[at(st, m)] = x;
        }
        wb = wbn;
    }
}

int qft_reg_tile_bits(qgpu_prec prec) {
    return prec == QGPU_C64 ? RegShape<float>::EB : RegShape<double>::EB;
}

template <typename R>
static void reg_launch(qgpu_ctx* ctx, const void* in, void* out, const QftRegPlan& p) {
    using C = Cplx<R>;
    // 32-bit offsets when the state has fewer than 2^31 amplitudes
    const bool narrow = p.ntiles <= (uint64_t(1) << (31 - RegShape<R>::EB));
    const size_t sm = (size_t(1) << RegShape<R>::EB) * sizeof(C) +
                      ((size_t(1) << (p.M - 1)) + (size_t(p.M) << p.nz) + 4 * size_t(p.M)) * sizeof(double2) +
                      size_t(p.nround) * kThr * sizeof(uint16_t) + (2 * kThr + 2 * RegShape<R>::NR) * (narrow ? sizeof(uint32_t) : sizeof(uint64_t));
    // 16 CTAs per SM, several tiles each: 2.00 ms a 28-qubit pass; with 4 the
    // pass that reverses took 2.70 instead of 2.46 ms
    uint64_t blocks = uint64_t(grid_blocks(ctx, 16));
    if (p.ntiles < blocks) blocks = p.ntiles;
    using K = void (*)(const C*, C*, const QftRegPlan);
    const K kern = narrow ? (p.inverse ? K(k_qft_reg<R, true, uint32_t>) : K(k_qft_reg<R, false, uint32_t>))
                          : (p.inverse ? K(k_qft_reg<R, true, uint64_t>) : K(k_qft_reg<R, false, uint64_t>));
    ensure_smem(reinterpret_cast<const void*>(kern), sm);
    kern<<<unsigned(blocks), kThr, sm, ctx->stream>>>(static_cast<const C*>(in), static_cast<C*>(out), p);
    after_launch(ctx, "k_qft_reg");
}

void launch_qft_reg(qgpu_ctx* ctx, qgpu_prec prec, const void* in, void* out, const QftRegPlan& p) {
    if (p.ntiles == 0) return;
    if (prec == QGPU_C64) reg_launch<float>(ctx, in, out, p);
    else reg_launch<double>(ctx, in, out, p);
}

} // namespace qgpu
