// kernels_regtile32.cu -- complex64 runs of 1- and 2-qubit gates as tile passes
// whose tile lives in registers, many registers (states) per launch.
//
// The complex64 counterpart of kernels_regtile.cu (programs: reg_tiles.hpp);
// there is no FP32 matrix instruction at full precision, so gates run as
// separate FMAs on register slots: a 2-qubit gate costs 16 of them per
// amplitude, and the program trades lane and register slots (a shuffle and
// three selects per amplitude pair and word) to bring its bits there.
//
// What bounds it: issue (a 2-qubit gate is 256 FMAs of a thread's 16
// amplitudes, a swap 64 shuffles and selects) and, per pass, the tile's way in
// and out. 2^12 amplitudes over 256 threads at 80 registers leave three CTAs
// per SM; half of a 4 x 4 matrix is held in registers at a time to stay there.
// Measured on one B200 against tiles kept in shared memory (a trip through it
// for every three bits): 330 gates gate by gate on 14 / 17 / 20 / 22 qubits
// 0.81 / 0.94 / 1.04 / 2.21 -> 0.20 / 0.20 / 0.30 / 1.14 ms, three layers on 24
// and 27 qubits 3.14 and 24.1 -> 1.32 and 11.5 ms. Per pass over 2^20
// amplitudes of 2^26: 3.5 us in and out, 0.67 us per 2-qubit gate (0.46 at the
// FP32 peak), 0.38 us per 1-qubit gate, 0.4 us per swap. Swaps pick with a logic
// operation: as selects on a predicate one took 0.68 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.hpp"
#include "reg_tiles.hpp"
#include "regtile32.cuh"

namespace qgpu {

// Tiles of one register (MANY = false: `one`) or of many (insts).
template <int NR, int NTMAX, int MINB, bool MANY>
__global__ void __launch_bounds__(NTMAX, MINB)
    k_reg_tile32(const RtInst* __restrict__ insts, const __grid_constant__ RtInst one, int ninst,
                 uint32_t ntiles, int T, int L) {
    extern __shared__ __align__(16) unsigned char rt_raw[];
    float2* const tile = reinterpret_cast<float2*>(rt_raw);
    const int nhi = T - L;
    uint64_t* const hioff = reinterpret_cast<uint64_t*>(rt_raw + (sizeof(float2) << T));
    unsigned char* const prog = reinterpret_cast<unsigned char*>(hioff) +
                                ((sizeof(uint64_t) << nhi) + 15) / 16 * 16;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    // a contiguous range of tiles, so that a CTA changes registers rarely
    const uint32_t t0 = uint32_t(uint64_t(ntiles) * blockIdx.x / gridDim.x);
    const uint32_t t1 = uint32_t(uint64_t(ntiles) * (blockIdx.x + 1) / gridDim.x);
    int ri = 0;
    if constexpr (MANY) {
        int hi = ninst - 1; // last register with first_tile <= t0
        while (ri < hi) {
            const int mid = (ri + hi + 1) >> 1;
            if (insts[mid].first_tile <= t0) ri = mid;
            else hi = mid - 1;
        }
    }
    int have = -1;
    const RtHead* const head = reinterpret_cast<const RtHead*>(prog);
    const RtOp* const ops = reinterpret_cast<const RtOp*>(prog + kRtHeadBytes);
    for (uint32_t t = t0; t < t1; ++t) {
        RtInst I;
        if constexpr (MANY) {
            while (ri + 1 < ninst && insts[ri + 1].first_tile <= t) ++ri;
            I = insts[ri];
        } else {
            I = one;
        }
        if (have != ri) { // the register's tables (uniform over the CTA)
            have = ri;
            for (uint32_t i = tid * 16; i < I.blob_bytes; i += nt * 16) {
                const uint32_t a = uint32_t(__cvta_generic_to_shared(prog + i));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(I.blob + i)
                             : "memory");
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            for (uint32_t j = tid; j < (1u << nhi); j += nt) {
                uint64_t o = 0;
                for (int i = 0; i < nhi; ++i)
                    if ((j >> i) & 1u) o |= uint64_t(1) << head->hi[i];
                hioff[j] = o;
            }
            __syncthreads();
        }
        uint64_t base = uint64_t(t - I.first_tile) << L;
        for (int i = 0; i < nhi; ++i) {
            const uint64_t lo = (uint64_t(1) << head->hi[i]) - 1;
            base = ((base & ~lo) << 1) | (base & lo);
        }
        const uint32_t nel = 1u << T, low = (1u << L) - 1, nvalid = head->nvalid;
        for (uint32_t e = 2 * tid; e < nel; e += 2 * nt) {
            float2* const d = &tile[rt_swz32_dev(e)];
            if (e + 1 < nvalid) {
                const uint32_t a = uint32_t(__cvta_generic_to_shared(d));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(a),
                             "l"(I.psi + base + hioff[e >> L] + (e & low))
                             : "memory");
            } else {
                d[0] = e < nvalid ? I.psi[e] : make_float2(0.f, 0.f);
                d[1] = make_float2(0.f, 0.f);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        float2 v[1 << NR];
        const uint32_t nops = head->nops;
        const RtLayoutTab* const lays = reinterpret_cast<const RtLayoutTab*>(
            prog + kRtHeadBytes + (nops * sizeof(RtOp) + 15) / 16 * 16);
        const float4* const coef = reinterpret_cast<const float4*>(lays + head->nlay);
        rt32_load<NR>(v, tile, lays[0], T, lane, warp);
        for (uint32_t o = 0; o < nops; ++o)
            rt32_op<NR>(v, ops[o], lays, coef, tile, T, lane, warp, base);
        __syncwarp();
        rt32_store<NR>(v, tile, lays[head->nlay - 1], T, lane, warp);
        __syncthreads();
        for (uint32_t e = 2 * tid; e < nel; e += 2 * nt) {
            const float2* const s = &tile[rt_swz32_dev(e)];
            float2* const d = I.psi + base + hioff[e >> L] + (e & low);
            if (e + 1 < nvalid) *reinterpret_cast<float4*>(d) = *reinterpret_cast<const float4*>(s);
            else if (e < nvalid) *d = *s;
        }
        __syncthreads();
    }
}

template <typename K>
static void launch_one32(K kernel, qgpu_ctx* ctx, const RtInst* dinsts, const RtInst& one, int ninst,
                         uint32_t ntiles, int T, int L, int NR, uint32_t blob_max, cudaStream_t stream,
                         int per_sm) {
    const size_t smem = (sizeof(float2) << T) + ((sizeof(uint64_t) << (T - L)) + 15) / 16 * 16 + blob_max;
    if (smem > kRt32SmemMax)
        raise(QGPU_ERR_NOT_SUPPORTED, "qgpu_run_gates()", "tile above the shared memory");
    ensure_smem(reinterpret_cast<const void*>(kernel), kRt32SmemMax);
    per_sm = std::max(1, std::min(per_sm, int(232448 / (smem + 1024))));
    const uint32_t grid = std::min<uint32_t>(ntiles, uint32_t(ctx->num_sms) * uint32_t(per_sm));
    kernel<<<grid, 32u << (T - 5 - NR), smem, stream>>>(dinsts, one, ninst, ntiles, T, L);
    after_launch(ctx, "k_reg_tile32");
}

void launch_reg_pass32(qgpu_ctx* ctx, const RtInst* dinsts, const RtInst& one, int ninst,
                       uint32_t ntiles, int T, int L, int NR, uint32_t blob_max, cudaStream_t stream) {
    if (ninst <= 0 || ntiles == 0) return;
    blob_max = (blob_max + 15) / 16 * 16;
    auto go = [&](auto kernel, int per_sm) {
        launch_one32(kernel, ctx, dinsts, one, ninst, ntiles, T, L, NR, blob_max, stream, per_sm);
    };
    if (dinsts && NR == 4) go(k_reg_tile32<4, 256, 3, true>, 3);
    else if (dinsts) go(k_reg_tile32<2, 512, 2, true>, 2);
    else if (NR == 4) go(k_reg_tile32<4, 256, 3, false>, 3);
    else go(k_reg_tile32<2, 512, 2, false>, 2);
}

} // namespace qgpu
