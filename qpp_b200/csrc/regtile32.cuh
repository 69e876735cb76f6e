// regtile32.cuh -- the ops of complex64 register tile programs (reg_tiles.hpp)
// on a thread's 2^NR amplitudes.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "reg_tiles.hpp"

namespace qgpu {

__device__ __forceinline__ uint32_t rt_swz32_dev(uint32_t e) {
    uint32_t r = e >> 4, h = 0;
#pragma unroll
    for (int k = 0; k < 16; k += 3) h ^= r >> k;
    return e ^ ((h & 7u) << 1);
}

// The products that begin a gate's sums, with their rounding spelled out so that
// a gate gives the same bits in every kernel that a seeded shot may run in: of
// the imaginary part's two terms a.y b.x is rounded and a.x b.y fused in a 4 x 4
// (c32_mul), the other way round in a 2 x 2 (c32_mul2).
__device__ __forceinline__ float2 c32_mul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 c32_mul2(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.y, b.x, __fmul_rn(a.x, b.y)));
}
__device__ __forceinline__ float2 c32_fma(float2 a, float2 b, float2 c) {
    c.x = fmaf(a.x, b.x, c.x);
    c.x = fmaf(-a.y, b.y, c.x);
    c.y = fmaf(a.x, b.y, c.y);
    c.y = fmaf(a.y, b.x, c.y);
    return c;
}

// A thread's position of register 0 in a layout, and the register slots'
// contributions.
template <int NR>
__device__ __forceinline__ uint32_t rt32_pos(const RtLayoutTab& lay, int T, int lane, int warp,
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
__device__ __forceinline__ uint32_t rt32_at(uint32_t b, const uint32_t (&ro)[NR], int j) {
#pragma unroll
    for (int k = 0; k < NR; ++k)
        if (j & (1 << k)) b ^= ro[k];
    return b;
}

template <int NR>
__device__ __forceinline__ void rt32_load(float2 (&v)[1 << NR], const float2* tile,
                                          const RtLayoutTab& lay, int T, int lane, int warp) {
    uint32_t ro[NR];
    const uint32_t b = rt32_pos<NR>(lay, T, lane, warp, ro);
#pragma unroll
    for (int j = 0; j < (1 << NR); ++j) v[j] = tile[rt32_at<NR>(b, ro, j)];
}

template <int NR>
__device__ __forceinline__ void rt32_store(const float2 (&v)[1 << NR], float2* tile,
                                           const RtLayoutTab& lay, int T, int lane, int warp) {
    uint32_t ro[NR];
    const uint32_t b = rt32_pos<NR>(lay, T, lane, warp, ro);
#pragma unroll
    for (int j = 0; j < (1 << NR); ++j) tile[rt32_at<NR>(b, ro, j)] = v[j];
}

template <bool CTRL>
__device__ __forceinline__ void rt32_put(float2& v, float2 r, bool ok) {
    if constexpr (CTRL) {
        v.x = ok ? r.x : v.x;
        v.y = ok ? r.y : v.y;
    } else {
        v = r;
    }
}

// 4 x 4 (row-major, two entries per float4; COL: column-major) on register slots
// A < B: rows 0 and 1 of every group first, then rows 2 and 3, so that half the
// matrix is held at a time.
template <int NR, int A, int B, bool CTRL, bool COL = false>
__device__ __forceinline__ void rt32_g2(float2 (&v)[1 << NR], const float4* m, bool lane_ok,
                                        uint32_t rmask, uint32_t rval) {
    if constexpr (B < NR) {
        constexpr int G = 1 << (NR - 2);
        float2 o[G][2];
        auto base = [](int g) { // zeros inserted at A and B
            int j = ((g >> A) << (A + 1)) | (g & ((1 << A) - 1));
            return ((j >> B) << (B + 1)) | (j & ((1 << B) - 1));
        };
        float2 c[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 e = m[COL ? half + 2 * k : 4 * half + k];
                c[COL ? 0 : k >> 1][COL ? k : 2 * (k & 1)] = make_float2(e.x, e.y);
                c[COL ? 1 : k >> 1][COL ? k : 2 * (k & 1) + 1] = make_float2(e.z, e.w);
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int j = base(g);
                const float2 x0 = v[j], x1 = v[j | 1 << A], x2 = v[j | 1 << B], x3 = v[j | 1 << A | 1 << B];
                float2 r[2];
#pragma unroll
                for (int row = 0; row < 2; ++row) {
                    r[row] = c32_mul(c[row][0], x0);
                    r[row] = c32_fma(c[row][1], x1, r[row]);
                    r[row] = c32_fma(c[row][2], x2, r[row]);
                    r[row] = c32_fma(c[row][3], x3, r[row]);
                }
                if (half == 0) {
                    o[g][0] = r[0];
                    o[g][1] = r[1];
                    continue;
                }
                const bool ok = lane_ok && (j & rmask) == rval;
                rt32_put<CTRL>(v[j], o[g][0], ok);
                rt32_put<CTRL>(v[j | 1 << A], o[g][1], ok);
                rt32_put<CTRL>(v[j | 1 << B], r[0], ok);
                rt32_put<CTRL>(v[j | 1 << A | 1 << B], r[1], ok);
            }
        }
    }
}

template <int NR, int A, bool CTRL, bool COL = false>
__device__ __forceinline__ void rt32_g1(float2 (&v)[1 << NR], const float4* m, bool lane_ok,
                                        uint32_t rmask, uint32_t rval) {
    if constexpr (A < NR) {
        const float4 m0 = m[0], m1 = m[1];
        const float2 e0 = make_float2(m0.x, m0.y), e1 = make_float2(m0.z, m0.w);
        const float2 e2 = make_float2(m1.x, m1.y), e3 = make_float2(m1.z, m1.w);
        const float2 a00 = e0, a01 = COL ? e2 : e1, a10 = COL ? e1 : e2, a11 = e3;
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) {
            if (j & (1 << A)) continue; // compile-time
            const int j1 = j | (1 << A);
            const float2 r0 = c32_fma(a01, v[j1], c32_mul2(a00, v[j]));
            const float2 r1 = c32_fma(a11, v[j1], c32_mul2(a10, v[j]));
            const bool ok = lane_ok && (j & rmask) == rval;
            rt32_put<CTRL>(v[j], r0, ok);
            rt32_put<CTRL>(v[j1], r1, ok);
        }
    }
}

// Bits of a where m is set, of b elsewhere (one three-input logic operation).
__device__ __forceinline__ float rt32_sel(uint32_t m, float a, float b) {
    return __uint_as_float((__float_as_uint(a) & m) | (__float_as_uint(b) & ~m));
}

// up: all ones in lanes whose bit is set
template <int NR, int B>
__device__ __forceinline__ void rt32_swap(float2 (&v)[1 << NR], uint32_t up, int xm) {
    if constexpr (B < NR) {
#pragma unroll
        for (int j = 0; j < (1 << NR); ++j) {
            if (j & (1 << B)) continue; // compile-time
            float2 &v0 = v[j], &v1 = v[j | (1 << B)];
            // a lane with bit 0 gives v1 and takes its partner's v0 there
            const float sx = __shfl_xor_sync(0xffffffffu, rt32_sel(up, v0.x, v1.x), xm);
            const float sy = __shfl_xor_sync(0xffffffffu, rt32_sel(up, v0.y, v1.y), xm);
            v0 = make_float2(rt32_sel(up, sx, v0.x), rt32_sel(up, sy, v0.y));
            v1 = make_float2(rt32_sel(up, v1.x, sx), rt32_sel(up, v1.y, sy));
        }
    }
}

template <int NR, bool CTRL>
__device__ __forceinline__ void rt32_gate(float2 (&v)[1 << NR], const RtOp& op, const float4* m,
                                          bool ok, uint32_t rm, uint32_t rv) {
    if (op.type == kRtG2) {
        switch (op.a * 4 + op.b) {
            case 1: rt32_g2<NR, 0, 1, CTRL>(v, m, ok, rm, rv); break;
            case 2: rt32_g2<NR, 0, 2, CTRL>(v, m, ok, rm, rv); break;
            case 3: rt32_g2<NR, 0, 3, CTRL>(v, m, ok, rm, rv); break;
            case 6: rt32_g2<NR, 1, 2, CTRL>(v, m, ok, rm, rv); break;
            case 7: rt32_g2<NR, 1, 3, CTRL>(v, m, ok, rm, rv); break;
            default: rt32_g2<NR, 2, 3, CTRL>(v, m, ok, rm, rv); break;
        }
        return;
    }
    switch (op.a) {
        case 0: rt32_g1<NR, 0, CTRL>(v, m, ok, rm, rv); break;
        case 1: rt32_g1<NR, 1, CTRL>(v, m, ok, rm, rv); break;
        case 2: rt32_g1<NR, 2, CTRL>(v, m, ok, rm, rv); break;
        default: rt32_g1<NR, 3, CTRL>(v, m, ok, rm, rv); break;
    }
}

// One op (any but kRtTrade); every thread of the CTA calls it with the same op. base:
// the index bits outside the tile.
template <int NR>
__device__ __forceinline__ void rt32_op(float2 (&v)[1 << NR], const RtOp& op, const RtLayoutTab* lays,
                                        const float4* coef, float2* tile, int T, int lane, int warp,
                                        uint64_t base) {
    const int type = op.type;
    if (type <= kRtG1L) {
        const float4* const m = coef + op.coef;
        if (op.ctrl) {
            if ((base & op.gmask) != op.gval || (warp & op.wmask) != op.wval) return;
            rt32_gate<NR, true>(v, op, m, (lane & op.lmask) == op.lval, op.rmask, op.rval);
        } else {
            rt32_gate<NR, false>(v, op, m, true, 0, 0);
        }
    } else if (type == kRtSwap) {
        const int xm = 1 << op.a;
        const uint32_t up = (lane & xm) ? ~0u : 0u;
        switch (op.b) {
            case 0: rt32_swap<NR, 0>(v, up, xm); break;
            case 1: rt32_swap<NR, 1>(v, up, xm); break;
            case 2: rt32_swap<NR, 2>(v, up, xm); break;
            default: rt32_swap<NR, 3>(v, up, xm); break;
        }
    } else {
        // a warp writes the positions it read at the last layout (swaps stay
        // inside a warp), so one barrier orders the writes before the reads
        __syncwarp();
        rt32_store<NR>(v, tile, lays[op.coef], T, lane, warp);
        __syncthreads();
        rt32_load<NR>(v, tile, lays[op.coef + 1], T, lane, warp);
    }
}

} // namespace qgpu
