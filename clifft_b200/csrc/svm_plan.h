// Fused blocks formed on the host. Which opcodes share one pass over the
// statevector depends only on the program (opcodes, axes, active ranks) and on
// the tile geometry, so the blocks of a program are planned once per geometry
// and a shot only fills in what its Pauli frame decides: the coefficients.
#pragma once

#include <cstdint>
#include <vector>

namespace cgpu {

// One fused block: instructions [pc, pc + n_instr) of the device stream.
struct BlockPlan {
    uint64_t F;          // tile axes
    uint64_t C;          // the other axes of the 2^kk amplitudes
    uint32_t pc;         // 0xffffffff closes the list
    uint32_t n_instr;
    uint32_t first_mop;  // its micro-ops in the plan's PlanOp array
    uint32_t n_mops;     // with a terminating measurement's own (SWAP, H)
    uint32_t n_body;     // without them
    uint32_t r;          // log2 of a tile's contiguous runs
    uint32_t kk;         // active rank while the block streams
    uint32_t skip;       // run-index bits of the axes the block creates (not loaded)
    uint32_t n_fresh;    // how many axes it creates
    uint32_t fresh_local;  // their tile-local bits
    uint32_t term_kind;  // measurement ending it: 0 none, 1 diagonal, 2 X basis, 3 X basis with a fused swap
    uint32_t term_pc;
    uint32_t red_local;  // the measured axis is a tile axis ...
    uint32_t red_bit;    // ... with this local bit, or its tile-global bit
    uint32_t single;     // the state is one tile, already in shared memory
    uint32_t pad;
};
static_assert(sizeof(BlockPlan) == 80 && sizeof(BlockPlan) % 16 == 0, "copied in 16-byte words");

// The frame-independent part of a micro-op, laid out like the head of
// MicroOpT, then what an index run keeps in unused coefficient slots: the
// rows of a diagonal op and (first op of a run) the columns of the final map.
struct PlanOp {
    uint8_t kind, a, b, flags;
    uint32_t req, par, pad;
    uint64_t greq, gpar;
    uint16_t row[3];
    uint8_t n_rows, pad2;
    uint16_t cols[12];
};
static_assert(sizeof(PlanOp) == 64, "copied in 16-byte words");

struct PlanGeometry {
    uint32_t bits;     // log2 of the amplitudes per tile
    uint32_t max_ops;  // micro-op slots per block (1: one opcode per pass)
    bool cta;          // a CTA per shot (scalar opcodes between blocks run on its control warp)
    bool team;         // ... which keeps states of at most one tile in shared memory
};

struct PlanSet {
    std::vector<BlockPlan> blocks;  // by pc, closed by a block with pc = 0xffffffff
    std::vector<PlanOp> ops;
};

// The blocks of the device instruction stream `code` (32 bytes each).
PlanSet plan_blocks(const uint8_t* code, uint32_t n_code, const PlanGeometry& g);

}  // namespace cgpu
