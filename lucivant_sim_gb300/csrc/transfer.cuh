// Host lowering of real64 register blocks: a trace-preserving Pauli-transfer operator of one qubit as
// shears between pairs of coefficients (tile.cuh rb_transfer), its scales merged into the block's
// diagonals (transfer.cu).
#pragma once

#include <cstdint>
#include <vector>

#include "lower.cuh"
#include "program.cuh"

namespace lsg {

// Move the outer rotation of the last two coefficients of every such operator (a rotation about Z, with
// the digits in the order I, Z, X, Y) through the renames and diagonals that let it pass into the next
// one on the same register bits. The operators then read entries appended to `pool` (and `low`, as
// move_outer_factors).
void move_outer_rotations(Plan& plan, int64_t batch, std::vector<double>& pool, std::vector<double>& low, Choices& form);

struct TransferItem {
    int op = -1;     // an operator kept as it is: its index in plan.ops; -1: made here
    int mask = -1;   // transfer operators: kTr* parts some member has, and positions P0 + 4 * P1; -1: a diagonal
    int pos[2] = {0, 0};
    std::vector<double> v;  // members x 2^u, or members x kTransferLen
};

// Entries of a lowered operator per member: parts, V (2), W (2), S (2), shift (3), then the rows of a
// member that keeps the dense form (12, 16-byte aligned).
constexpr int kTransferLen = 22;

// False when the block would not take fewer operations. members: 1 when all data are shared.
bool lower_transfer_block(const Plan& plan, const PassDesc& pd, const BlockDesc& blk, int64_t batch, const Pool& pool,
                          Choices& form, std::vector<TransferItem>* items, int64_t* members);

}  // namespace lsg
