// tile_gates.hpp -- planning and execution of gate runs as tile passes
// (tile_gates.cpp, reg_tiles.cpp).
#pragma once

#include <complex>
#include <utility>
#include <vector>

#include "internal.hpp"
#include "kernels.hpp"

namespace qgpu {

struct Step;

// One 1- or 2-qubit gate of a qubit ket: state bits b0 (and b1 for op 2; the
// matrix's row index is 2 * b(b0) + b(b1)), controls as (state bit, value),
// the matrix column-major.
struct GateDesc {
    int op = 1;
    int b0 = 0, b1 = 0;
    std::vector<std::pair<int, int>> ctrl;
    cd A[16];
};

// Appends the gates of step `st` on an nbits-qubit ket and returns true, or
// returns false (appending nothing) when the step is not a 1- or 2-qubit
// unitary, fan or controlled gate.
bool gate_desc_of(const Step& st, int nbits, std::vector<GateDesc>& out);
// Splits `gates` (in order) into tile passes of at most Tmax tile bits: the
// low min(nbits, 5) state bits and the targets above them; each pass into
// sweeps of consecutive gates on at most three tile bits. `dev` gets one
// entry per gate with tile-local bits, `sweeps` the sweeps, `mats` the
// row-major matrices.
void plan_gate_tiles(const std::vector<GateDesc>& gates, int nbits, int Tmax,
                     std::vector<TilePassParams>& passes, std::vector<TileGate>& dev,
                     std::vector<TileSweep>& sweeps, std::vector<cd>& mats);
// The gates reordered for fewer tile passes and sweeps (list scheduling):
// every gate still follows the earlier gates it shares a bit with (target or
// control), so the product is the same up to rounding, but each pass takes
// every ready gate whose targets fit the tile, those that extend the current
// sweep first. For forms that do not promise the gate-by-gate arithmetic.
std::vector<GateDesc> schedule_gates(const std::vector<GateDesc>& gates, int nbits, int Tmax);
// Largest tile (bits) for this context: kRtMaxTile, or qgpu_ctx_set_tile_bits's
// where that is less.
int tile_bits_max(const qgpu_ctx* ctx);
// Uploads P's tables and launches its passes on s (stream order; the tile in
// registers, reg_tiles.hpp).
struct RegProgram;
void run_reg_program(qgpu_state* s, const RegProgram& P);
// Plans the gates into P, each pass launched as soon as it is planned.
void plan_and_run_reg(qgpu_state* s, const std::vector<GateDesc>& gates, int Tmax, RegProgram& P);
// Runs `gates` on the qubit ket s as planned tile passes (stream order).
void run_tiled_gates(qgpu_state* s, const std::vector<GateDesc>& gates);

// A piece of a fused complex128 ket plan: a run of gate descriptors for the
// tile passes (step < 0; possibly empty), or one step run as it is.
struct TiledRun {
    std::vector<GateDesc> gates;
    int64_t step = -1;
};
// The circuit's fused plan (blocks of <= 2 qubits, c->plan) and its unfused
// steps, in circuit order, as tile-pass runs and steps.
void tiled_runs(const qgpu_circuit* c, std::vector<TiledRun>& out);

} // namespace qgpu
