// reg_tiles.h — register passes: tiled passes over a state whose gates all
// fit a thread's registers (1- and 2-qubit gates, permutations, diagonals of
// any width, with controls).  Planned on the host here, run by reg_tiles.cu.
#pragma once

#include <cstdint>
#include <vector>

#include "yao_internal.h"

namespace yao {

// A segment: the ops [op_begin, op_end) applied while each thread holds the
// 2^RB amplitudes that differ in RB tile positions.  sorted[]: those
// positions ascending; order[i]: the position that amplitude-index bit i
// stands for.
struct RSeg {
    int32_t op_begin, op_end;
    int8_t sorted[4];
    int8_t order[4];
};

// One op, 32 bytes, read by every thread as two 16-byte words.
//   head: code in bits 0..7, amplitude mask in bits 16..31 (bit j: the pair,
//         group or amplitude whose first member is amplitude j takes part)
//   coef: first coefficient (complex numbers from the pass's first)
//   ctl:  controls on the thread's own tile positions: mask in bits 0..15,
//         value in bits 16..31
//   gmask / gval: controls outside the tile, as bits of the tile's number
//   sel0, sel1: a diagonal's targets outside the registers, lowest entry bit
//         first, 6 bits each (five in sel0, one in sel1): 0..15 a tile
//         position, 16.. a bit of the tile's number; their count in bits
//         8..15 of sel1
//   sign: 1-qubit matrices (never controlled): pairs whose second member is
//         negated first (a CZ that joined the matrix): always (bits 0..15),
//         and where the controls match (bits 16..31)
struct ROp {
    uint32_t head, coef, ctl, gmask, gval, sel0, sel1, sign;
};
static_assert(sizeof(ROp) == 32 && sizeof(RSeg) == 16, "read as 16-byte words");

enum RCode : uint32_t {
    // + position: a 2 x 2 matrix [[a, b], [c, d]] on every pair
    RC_DENSE1 = 0,   // complex
    RC_REAL1 = 4,    // real: two coefficients, a + i b and c + i d
    RC_RCOL1 = 8,    // a, c real: a + i c, b, d
    RC_RROW1 = 12,   // a, b real: a + i b, c, d
    RC_MASKED1 = 16, // + position: a complex 2 x 2 matrix on the masked pairs
    RC_X = 20,       // + position: swaps the masked pairs
    RC_PHASE1 = 24,  // + position: the amplitudes with that bit set times one coefficient
    RC_DENSE2 = 28,  // + pair (positions 2 pair, 2 pair + 1), masked
    RC_SWAP = 30,    // + pair, masked
    RC_PHASE = 32,   // the masked amplitudes times one coefficient
    RC_DIAG = 33,    // the masked amplitudes, each times its own coefficient
    RC_NEG = 34,     // the masked amplitudes times -1
    RC_LAYER = 35,   // amplitudes 1 to 15 times the coefficients from sel0 (~0: no such product), then
                     // REAL1 ops without pair signs on positions 0 to 3: this op and the next three
    // density-matrix steps
    RC_CHAN1 = 36,   // + pair: a 1-qubit Kraus sum; sel0: operators, three coefficients each (exact passes)
    RC_CHAN2 = 38,   // a 2-qubit Kraus sum; sel0: operators, five coefficients each (exact passes)
    RC_PAULI2 = 39,  // four real 4 x 4 matrices (not in exact passes)
    RC_REAL2 = 40    // + pair: a real 4 x 4 matrix with a phase a row (sel0 = 0) or a column (1)
};

struct RegPass {
    int tbits = 0, rb = 0;
    int8_t tb[16] = {0};
    uint64_t ntiles = 0;
    std::vector<RSeg> segs;
    std::vector<ROp> ops;
    std::vector<Cx> coef;
    size_t blob_off = 0, blob_bytes = 0;  // in the plan's packed blob
};

struct RegPlan {
    std::vector<RegPass> passes;
    std::vector<unsigned char> blob;  // every pass's segments | ops | coefficients
};

// Whether every gate can run in registers (dense gates on at most 2 qubits).
bool reg_supported(const std::vector<LGate>& prog, uint32_t nbits);
// The FUSED program for register passes (host, FP64): 1-qubit gates between
// the gates that touch their qubit are multiplied together and written as
// phase . real rotation . phase, a CNOT between two rotations of its target
// becomes a CZ (its Hadamards join the rotations), and phases move past
// controls and diagonals to the next rotation.  Other gates are kept.
void split_single_qubit(const std::vector<LGate>& prog, uint32_t nbits, std::vector<LGate>& out);
// Tiles that fill the GPU twice over (148 SMs; a constant, so that a program
// has one plan wherever it is made).
constexpr uint64_t kManyTiles = 2 * 148;
// Passes over 2^tbits-amplitude tiles.  exact: program order, except that
// permutations (X, SWAP, with controls) may move past gates on other qubits,
// which changes no bit of the result; otherwise any gate may.
// batch_tiles: the tiles of all registers that run together (0: this one).
void reg_plan(const std::vector<LGate>& prog, uint32_t nbits, int32_t precision, int tbits, bool exact, RegPlan& out,
              uint64_t batch_tiles = 0);
// Queues passes first, first + step, ... of the plan on the context's stream.
// *queued: whether an error left some of them queued.
int reg_launch(Ctx* ctx, void* st, uint32_t nbits, int32_t precision, bool exact, const RegPlan& plan, size_t first,
               size_t step, bool* queued = nullptr);

// Runs plan c on register c for all c, and waits.  Every plan has the same
// number of amplitudes a thread (planned with the same batch_tiles).
int reg_batch(Ctx* ctx, const std::vector<RegPlan>& plans, const std::vector<Reg*>& regs, bool exact);

// Fusion into blocks of at most 2 qubits (sv_tiles.cu); density-matrix steps
// on two qubits are kept.
void fuse_two_qubit(const std::vector<LGate>& prog, uint32_t nbits, std::vector<LGate>& out);
// A program with each gate's own arithmetic in program order (the PLAIN
// form): runs of gates as exact register passes where that is faster, else
// one launch a gate; the results are the same bits either way.  Wide gates,
// complex64 and runs under stream capture: one launch a gate.
int plain_run(Ctx* ctx, Reg* r, const std::vector<LGate>& prog);

}  // namespace yao
