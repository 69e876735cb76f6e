// kernels_regtile.cu -- complex128 runs of 1- and 2-qubit gates as tile passes
// whose tile lives in registers.
//
// Replaces, for runs of gates on a qubit ket, the one-pass-per-gate loops of
// include/qpp/internal/kernels/qubit/apply.hpp:57-265 (apply_psi_1q/2q) and
// apply_ctrl.hpp:63-265. A CTA takes a tile of 2^T amplitudes (the L lowest
// state bits and T - L others), reads it into shared memory, spreads it over
// its registers (slots, reg_tiles.hpp), runs the pass's program and writes it
// back: one read and one write of the state per pass.
//
// 2-qubit gates run on the FP64 matrix instruction mma.m8n8k4: eight groups of
// four amplitudes are the 8 x 4 operand (real parts, then imaginary parts),
// the gate as a real 4 x 8 matrix the other. Its fragment layouts coincide:
// lane l holds amplitude l & 3 of group l >> 2 before and after, so a gate
// needs its two bits in lane slots 0 and 1 and nothing else moves. The
// program brings bits there by trading lane and register slots (shuffles) and,
// when a bit sits in a warp slot, through shared memory.
//
// What bounds it: the FP64 pipe (36.9 TFLOP/s measured for the matrix
// instruction, 30-33 for separate FMAs) plus the shuffles, and per pass the
// tile's way in and out. Why this split: 2^12 amplitudes over 256 threads (16
// in registers, 9 of 12 bits inside a warp) leave two CTAs per SM, one loading
// or storing while the other computes, and a layout change through shared
// memory is needed once in several gates; a tile kept in shared memory, with a
// trip through it for every three bits, ran at 28% of the FP64 pipe. Measured
// on one B200 against that form: 1100 gates on 2^20 amplitudes gate by gate
// 2.96 -> 1.60 ms, merged into 2-qubit blocks 1.40 -> 0.95 ms, 126 gates on
// 2^28 amplitudes 88.4 -> 43.1 ms. Per pass over 2^20 amplitudes: about 6 us in
// and out, 1.1 us per 2-qubit gate (the pipe's time), 0.8 or 1.2 us per 1-qubit
// gate on a register or lane slot, 0.33 us per swap or permutation, 1.6 us per
// layout change.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"
#include "reg_tiles.hpp"

namespace qgpu {

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

__device__ __forceinline__ uint32_t rt_swz_dev(uint32_t e) {
    uint32_t r = e >> 3, h = 0;
#pragma unroll
    for (int k = 0; k < 16; k += 3) h ^= r >> k;
    return e ^ (h & 7u);
}

template <bool CTRL>
__device__ __forceinline__ void rt_put(double2& v, double x, double y, bool ok) {
    if constexpr (CTRL) {
        v.x = ok ? x : v.x;
        v.y = ok ? y : v.y;
    } else {
        v.x = x;
        v.y = y;
    }
}

template <int NR, bool CTRL>
__device__ __forceinline__ void rt_g2(double2 (&v)[1 << NR], double2 c, bool lane_ok, uint32_t rmask,
                                      uint32_t rval) {
#pragma unroll
    for (int j = 0; j < (1 << NR); ++j) {
        double d0 = 0.0, d1 = 0.0;
        dmma(d0, d1, v[j].x, c.x);
        dmma(d0, d1, v[j].y, c.y);
        rt_put<CTRL>(v[j], d0, d1, lane_ok && (j & rmask) == rval);
    }
}

template <int NR, int A, bool CTRL>
__device__ __forceinline__ void rt_g1r(double2 (&v)[1 << NR], const double2* m, bool lane_ok,
                                       uint32_t rmask, uint32_t rval) {
    if constexpr (A < NR) {
        const double2 a00 = m[0], a01 = m[1], a10 = m[2], a11 = m[3];
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) {
            if (j & (1 << A)) continue; // compile-time
            const int j1 = j | (1 << A);
            const double2 r0 = cfma(a01, v[j1], cmul(a00, v[j]));
            const double2 r1 = cfma(a11, v[j1], cmul(a10, v[j]));
            const bool ok = lane_ok && (j & rmask) == rval;
            rt_put<CTRL>(v[j], r0.x, r0.y, ok);
            rt_put<CTRL>(v[j1], r1.x, r1.y, ok);
        }
    }
}

// own and other: the matrix entries on this lane's and its partner's amplitude
template <int NR, bool CTRL>
__device__ __forceinline__ void rt_g1l(double2 (&v)[1 << NR], double2 own, double2 other, int xm,
                                       bool lane_ok, uint32_t rmask, uint32_t rval) {
#pragma unroll
    for (int j = 0; j < (1 << NR); ++j) {
        double2 p;
        p.x = __shfl_xor_sync(0xffffffffu, v[j].x, xm);
        p.y = __shfl_xor_sync(0xffffffffu, v[j].y, xm);
        const double2 r = cfma(other, p, cmul(own, v[j]));
        rt_put<CTRL>(v[j], r.x, r.y, lane_ok && (j & rmask) == rval);
    }
}

template <int NR, int B>
__device__ __forceinline__ void rt_swap(double2 (&v)[1 << NR], bool up, int xm) {
    if constexpr (B < NR) {
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) {
            if (j & (1 << B)) continue; // compile-time
            double2 &v0 = v[j], &v1 = v[j | (1 << B)];
            // a lane with bit 0 gives v1 and takes its partner's v0 there
            double2 s;
            s.x = up ? v0.x : v1.x;
            s.y = up ? v0.y : v1.y;
            s.x = __shfl_xor_sync(0xffffffffu, s.x, xm);
            s.y = __shfl_xor_sync(0xffffffffu, s.y, xm);
            v0.x = up ? s.x : v0.x;
            v0.y = up ? s.y : v0.y;
            v1.x = up ? v1.x : s.x;
            v1.y = up ? v1.y : s.y;
        }
    }
}

// A thread's position of register 0 in a layout, and the register slots'
// contributions.
template <int NR>
__device__ __forceinline__ uint32_t rt_pos(const RtLayoutTab& lay, int T, int lane, int warp,
                                           uint32_t (&ro)[NR]) {
    uint32_t b = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i) b ^= ((lane >> i) & 1) ? lay.img[NR + i] : 0u;
    for (int i = NR + 5; i < T; ++i) b ^= ((warp >> (i - NR - 5)) & 1) ? lay.img[i] : 0u;
#pragma unroll
    for (int k = 0; k < NR; ++k) ro[k] = lay.img[k];
    return b;
}

template <int NR>
__device__ __forceinline__ uint32_t rt_at(uint32_t b, const uint32_t (&ro)[NR], int j) {
#pragma unroll
    for (int k = 0; k < NR; ++k)
        if (j & (1 << k)) b ^= ro[k];
    return b;
}

template <int NR, int NTMAX, int MINB>
__global__ void __launch_bounds__(NTMAX, MINB)
    k_reg_tile(double2* __restrict__ psi, const __grid_constant__ RegPass p,
               const unsigned char* __restrict__ blob) {
    extern __shared__ __align__(16) unsigned char rt_raw[];
    double2* const tile = reinterpret_cast<double2*>(rt_raw);
    const int nhi = p.T - p.L;
    uint64_t* const hioff = reinterpret_cast<uint64_t*>(rt_raw + (sizeof(double2) << p.T));
    unsigned char* const prog = reinterpret_cast<unsigned char*>(hioff) +
                                ((sizeof(uint64_t) << nhi) + 15) / 16 * 16;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t i = tid * 16; i < p.blob_bytes; i += nt * 16) {
        const uint32_t a = uint32_t(__cvta_generic_to_shared(prog + i));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(blob + i) : "memory");
    }
    cp_async_commit();
    for (uint32_t j = tid; j < (1u << nhi); j += nt) {
        uint64_t o = 0;
        for (int i = 0; i < nhi; ++i)
            if ((j >> i) & 1u) o |= uint64_t(1) << p.hi[i];
        hioff[j] = o;
    }
    const RtOp* const ops = reinterpret_cast<const RtOp*>(prog);
    const RtLayoutTab* const lays = reinterpret_cast<const RtLayoutTab*>(
        prog + (p.nops * sizeof(RtOp) + 15) / 16 * 16);
    const double2* const coef = reinterpret_cast<const double2*>(lays + p.nlay);
    __syncthreads(); // hioff
    const uint32_t nel = 1u << p.T, low = (1u << p.L) - 1;
    for (uint64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
        // tile number -> base offset: zeros inserted at every tile bit
        uint64_t base = t << p.L;
        for (int i = 0; i < nhi; ++i) {
            const uint64_t lo = (uint64_t(1) << p.hi[i]) - 1;
            base = ((base & ~lo) << 1) | (base & lo);
        }
        for (uint32_t e = tid; e < nel; e += nt) {
            if (e < p.nvalid) cp_async_elem(&tile[rt_swz_dev(e)], &psi[base + hioff[e >> p.L] + (e & low)]);
            else tile[rt_swz_dev(e)] = make_double2(0.0, 0.0);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        double2 v[1 << NR];
        uint32_t ro[NR];
        uint32_t b = rt_pos<NR>(lays[0], p.T, lane, warp, ro);
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) v[j] = tile[rt_at<NR>(b, ro, j)];
        for (uint32_t o = 0; o < p.nops; ++o) {
            const RtOp& op = ops[o];
            const int type = op.type;
            if (type <= kRtG1L) {
                const bool ctrl = op.ctrl != 0;
                uint32_t rm = 0, rv = 0;
                bool ok = true;
                if (ctrl) {
                    if ((base & op.gmask) != op.gval || (warp & op.wmask) != op.wval) continue;
                    rm = op.rmask;
                    rv = op.rval;
                    ok = (lane & op.lmask) == op.lval;
                }
                const double2* const m = coef + op.coef;
                if (type == kRtG2) {
                    const double2 c = m[lane];
                    if (ctrl) rt_g2<NR, true>(v, c, ok, rm, rv);
                    else rt_g2<NR, false>(v, c, true, 0, 0);
                } else if (type == kRtG1L) {
                    const int s = (lane >> op.a) & 1;
                    const double2 own = m[3 * s], other = m[1 + s];
                    if (ctrl) rt_g1l<NR, true>(v, own, other, 1 << op.a, ok, rm, rv);
                    else rt_g1l<NR, false>(v, own, other, 1 << op.a, true, 0, 0);
                } else if (ctrl) {
                    switch (op.a) {
                        case 0: rt_g1r<NR, 0, true>(v, m, ok, rm, rv); break;
                        case 1: rt_g1r<NR, 1, true>(v, m, ok, rm, rv); break;
                        case 2: rt_g1r<NR, 2, true>(v, m, ok, rm, rv); break;
                        default: rt_g1r<NR, 3, true>(v, m, ok, rm, rv); break;
                    }
                } else {
                    switch (op.a) {
                        case 0: rt_g1r<NR, 0, false>(v, m, true, 0, 0); break;
                        case 1: rt_g1r<NR, 1, false>(v, m, true, 0, 0); break;
                        case 2: rt_g1r<NR, 2, false>(v, m, true, 0, 0); break;
                        default: rt_g1r<NR, 3, false>(v, m, true, 0, 0); break;
                    }
                }
            } else if (type == kRtSwap) {
                const bool up = (lane >> op.a) & 1;
                const int xm = 1 << op.a;
                switch (op.b) {
                    case 0: rt_swap<NR, 0>(v, up, xm); break;
                    case 1: rt_swap<NR, 1>(v, up, xm); break;
                    case 2: rt_swap<NR, 2>(v, up, xm); break;
                    default: rt_swap<NR, 3>(v, up, xm); break;
                }
            } else if (type == kRtPerm) {
                int src = 0;
#pragma unroll
                for (int i = 0; i < 5; ++i) src |= ((lane >> i) & 1) << ((op.coef >> (3 * i)) & 7);
#pragma unroll
                for (int j = 0; j < (1 << NR); ++j) {
                    v[j].x = __shfl_sync(0xffffffffu, v[j].x, src);
                    v[j].y = __shfl_sync(0xffffffffu, v[j].y, src);
                }
            } else {
                // a warp writes the positions it read at the last layout (swaps
                // and permutations stay inside a warp), so one barrier orders
                // the writes before the new reads
                __syncwarp();
                b = rt_pos<NR>(lays[op.coef], p.T, lane, warp, ro);
#pragma unroll
                for (int j = 0; j < (1 << NR); ++j) tile[rt_at<NR>(b, ro, j)] = v[j];
                __syncthreads();
                b = rt_pos<NR>(lays[op.coef + 1], p.T, lane, warp, ro);
#pragma unroll
                for (int j = 0; j < (1 << NR); ++j) v[j] = tile[rt_at<NR>(b, ro, j)];
            }
        }
        __syncwarp();
        b = rt_pos<NR>(lays[p.nlay - 1], p.T, lane, warp, ro);
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) tile[rt_at<NR>(b, ro, j)] = v[j];
        __syncthreads();
        for (uint32_t e = tid; e < nel; e += nt)
            if (e < p.nvalid) psi[base + hioff[e >> p.L] + (e & low)] = tile[rt_swz_dev(e)];
        __syncthreads();
    }
}

size_t reg_pass_smem(const RegPass& p) {
    return (sizeof(double2) << p.T) + ((sizeof(uint64_t) << (p.T - p.L)) + 15) / 16 * 16 + p.blob_bytes;
}

template <typename K>
static void launch_one(K kernel, qgpu_ctx* ctx, void* data, const RegPass& p,
                       const unsigned char* blob, int per_sm) {
    const size_t smem = reg_pass_smem(p);
    ensure_smem(reinterpret_cast<const void*>(kernel), kRtSmemMax);
    const int nt = 32 << (p.T - 5 - p.NR);
    per_sm = std::max(1, std::min(per_sm, int(232448 / (smem + 1024))));
    const unsigned grid = unsigned(std::min<uint64_t>(p.ntiles, uint64_t(ctx->num_sms) * per_sm));
    kernel<<<grid, unsigned(nt), smem, ctx->stream>>>(static_cast<double2*>(data), p, blob);
    after_launch(ctx, "k_reg_tile");
}

void launch_reg_pass(qgpu_ctx* ctx, void* data, const RegPass& p, const unsigned char* blob) {
    if (reg_pass_smem(p) > kRtSmemMax)
        raise(QGPU_ERR_NOT_SUPPORTED, "qgpu_run_gates()", "tile above the shared memory");
    if (p.NR == 4) launch_one(k_reg_tile<4, 256, 2>, ctx, data, p, blob, 2);
    else launch_one(k_reg_tile<2, 512, 2>, ctx, data, p, blob, 2);
}

} // namespace qgpu
