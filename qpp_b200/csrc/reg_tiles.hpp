// reg_tiles.hpp -- tile passes with the tile held in registers (reg_tiles.cpp
// plans them on the host; kernels_regtile.cu runs the complex128 ones,
// kernels_regtile32.cu the complex64 ones).
#pragma once

#include <cstdint>
#include <functional>
#include <vector>

#include "tile_gates.hpp"

namespace qgpu {

// A tile of 2^T amplitudes is spread over one CTA: every tile bit sits in one
// slot, and slots [0, NR) number a thread's 2^NR registers, [NR, NR + 5) its
// lane, [NR + 5, T) its warp. A pass is a program of ops that every thread of
// the CTA runs in lockstep:
//   kRtG2      4 x 4. Complex128: on the bits in lane slots 0 and 1 (amplitude
//              index lane & 3), two FP64 matrix instructions per register.
//              Complex64: on the bits in register slots a < b (index bit a
//              plus 2 x bit b)
//   kRtG1R a   2 x 2 on the bit in register slot a
//   kRtG1L a   2 x 2 on the bit in lane slot a (its partner by a shuffle;
//              complex128 only)
//   kRtSwap    lane slot a and register slot b trade their bits
//   kRtPerm    lane slots permuted: slot i takes the bit of slot perm[i]
//              (coef = perm[i] << 3 i; complex128 only)
//   kRtLayout  every bit to a new slot through shared memory: written in
//              layout table coef, read back in table coef + 1
//   kRtTrade   register slots a < b trade their bits (complex64 programs planned
//              `ordered`; the kernels have no code for it)
enum : uint8_t {
    kRtG2 = 0, kRtG1R = 1, kRtG1L = 2, kRtSwap = 3, kRtPerm = 4, kRtLayout = 5, kRtTrade = 6
};

// Controls hold a gate to the amplitudes whose register, lane, warp and
// out-of-tile index bits under the masks equal the values.
struct RtOp {
    uint8_t type, a, b, ctrl;
    uint32_t coef; // gates: 16-byte units from the pass's coefficients
    uint8_t rmask, rval, lmask, lval, wmask, wval, pad[2];
    uint32_t pad2;
    uint64_t gmask, gval;
};
static_assert(sizeof(RtOp) == 40, "op size");

// The swizzled shared-memory position contributed by the bit of each slot
// (positions are XORs of these). Table 0 is the layout the tile is first read
// in, the last one the layout it is written back in.
struct RtLayoutTab {
    uint16_t img[16];
};

constexpr int kRtMaxTile = 12; // 64 KB of complex128, two CTAs per SM
constexpr int kRtMinTile = 7;  // 4 registers per lane, one warp
// Shared memory of a CTA (two per SM), and what a pass's program may take of
// it next to the largest tile and its offset table.
constexpr size_t kRtSmemMax = 112 * 1024;
constexpr size_t kRtBlobMax = 44 * 1024;
// Complex64: 32 KB tiles, three CTAs per SM.
constexpr size_t kRt32SmemMax = 75 * 1024;
constexpr size_t kRt32BlobMax = 38 * 1024;

struct RegPass {
    uint64_t ntiles;
    int T, L, NR;
    int hi[16];         // state bits of tile bits L .. T - 1, ascending
    uint32_t nvalid;    // amplitudes of the tile that exist (states below 2^kRtMinTile)
    uint32_t nops, nlay;
    uint32_t blob, blob_bytes; // the pass's ops, layouts and coefficients
    uint32_t ngates;
    int single;                // index of its only gate in RegProgram::single, or -1
};

// What a complex64 pass's tables begin with (its RegPass, on the device).
struct RtHead {
    uint32_t nops, nlay, nvalid;
    int32_t T, L, NR;
    int32_t hi[16];
};
static_assert(sizeof(RtHead) % 8 == 0, "head size");
constexpr size_t kRtHeadBytes = (sizeof(RtHead) + 15) / 16 * 16;

// One register's pass in a complex64 launch: tiles [first_tile, next one's) of
// the launch are its tiles.
struct RtInst {
    float2* psi;
    const unsigned char* blob;
    uint32_t first_tile, blob_bytes;
};

struct RegProgram {
    qgpu_prec prec = QGPU_C128;
    int nbits = 0;
    std::vector<RegPass> passes;
    std::vector<GateDesc> single; // passes of one uncontrolled gate
    std::vector<unsigned char> blob;
    bool trades = false; // holds kRtTrade: for the host model alone
};

// The tile shape for an nbits-qubit ket: T bits of which the L lowest state
// bits always belong to the tile, and 2^NR registers per thread.
void reg_tile_shape(qgpu_prec prec, int nbits, int Tmax, int& T, int& L, int& NR);
// Cuts the gates into passes and compiles each into its program (P.prec set
// by the caller). Gates on disjoint bits trade places (list scheduling); each
// bit's gates keep their order, so the product is the same up to rounding.
// `planned`, when given, is called after each pass with its tables in P.blob,
// so that the device can start while the host plans on. ordered (complex64):
// every 2-qubit product adds its four terms in the order of the matrix columns;
// such programs are not run (run_reg_program refuses them): the case that trades
// registers costs every other op about 30 moves to bring them back, 10% of a 2-qubit
// gate.
void plan_reg_program(const std::vector<GateDesc>& gates, int nbits, int Tmax, RegProgram& P,
                      const std::function<void(const RegPass&)>& planned = nullptr,
                      bool ordered = false);
// An upper bound of the program's bytes.
size_t reg_program_bytes(const std::vector<GateDesc>& gates);

// The fused complex128 tile form of a circuit, planned once: list-scheduled
// tile programs and the unfused steps between them, for the circuit's first
// nsteps steps and tiles of at most Tmax bits.
struct FusedTiles {
    uint64_t nsteps = 0;
    int Tmax = 0;
    std::vector<std::pair<int64_t, RegProgram>> runs; // first >= 0: that step as it is
};

// Swizzled shared-memory position of tile element e: 16-byte columns of the
// 128-byte rows XORed with the folded row number; a complex64 pair stays one
// column.
inline uint32_t rt_swz(uint32_t e) {
    uint32_t r = e >> 3, h = 0;
    for (int k = 0; k < 16; k += 3) h ^= r >> k;
    return e ^ (h & 7u);
}
inline uint32_t rt_swz32(uint32_t e) { return rt_swz(e >> 1) << 1 | (e & 1u); }

// Launches pass p (its tables at device address `blob`) on the ket at data.
void launch_reg_pass(qgpu_ctx* ctx, void* data, const RegPass& p, const unsigned char* blob);
// One launch over the complex64 passes of ninst registers (dinsts: a device
// table sorted by first_tile; null: the one register `one`), ntiles tiles in
// all, every pass of T tile bits and NR register slots and tables of at most
// blob_max bytes.
void launch_reg_pass32(qgpu_ctx* ctx, const RtInst* dinsts, const RtInst& one, int ninst,
                       uint32_t ntiles, int T, int L, int NR, uint32_t blob_max, cudaStream_t stream);

} // namespace qgpu
