// adj_group.cuh — the grouped passes of the adjoint sweep (adj_group.cu), used by adjoint.cu.
#pragma once

#include <vector>

#include "internal.cuh"
#include "plan.h"

namespace qgpu {

// One wire of a grouped pass: its index bit, the frame of its run's undo, and the partial rows of
// the sums Im <lambda| s |phi> it needs: X and Y after D1 of the frame, Z (-1: not needed).
struct AdjGroupWire {
    int bit;
    PauliFrame frame;
    int row[3];
};

// Widest tile of a pass.
int adj_group_tile_bits(int precision);

// One pass over phi and lambda (the handle's precision; complex128 in the resident float-pair
// layout) on the tile bits of `mask`, which hold every wire's bit. row_i: row of the sum over -I
// (-1: not needed). nb: the rows' length, the largest grid. *drift (0 at first): the
// relative change of both vectors' norms by the rounding of the rotations so far. Queued on the
// handle's stream.
int adj_group_pass(qgpu_handle* h, void* phi, void* lam, uint64_t mask,
                   const std::vector<AdjGroupWire>& wires, int row_i, double* partial, int nb,
                   double* drift);

}  // namespace qgpu
