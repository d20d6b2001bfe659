// Host lowering of complex register blocks to rounds (lower.cu): a round is one diagonal over the
// block's 2^u amplitudes followed by real plane rotations on its bits, each a pair of multiply-adds
// per amplitude (tile.cuh rb_round).
#pragma once

#include <complex>
#include <cstdint>
#include <vector>

#include "program.cuh"

namespace lsg {

// Move the outer factor of every one-bit operator of a planned complex program through the renames
// and diagonals that let it pass, into the next one-bit operator on the same register bit. The
// operators then read their matrices from entries appended to `pool` (complex entries as pairs), what
// the entries' rounding left over to `low`. Returns which operators (indexed like plan.ops) had their
// outer factor taken.
std::vector<char> move_outer_factors(Plan& plan, int64_t batch, std::vector<double>& pool, std::vector<double>& low);

// A program's data: `own` doubles of the caller's, then what move_outer_factors appended, with its `low`.
struct Pool {
    const double* data;
    const double* low;
    int64_t own;
};

// A lowered block: items in order, each a round (kT_ROUND: mask, diagonal, rotations) or an operator
// kept as it is (kKeepOp: index into plan.ops, its register-block code).
constexpr int kKeepOp = -2;
struct LoweredItem {
    int code = 0;
    int op = -1;
    int tmpl = 0;
    int mask = 0;  // rounds: bit P a rotation on block position P, bit 4 a diagonal
    std::vector<std::complex<double>> diag;  // members x 2^u
    std::vector<double> t, second;           // rounds: members x u rotations, (t, flip) or (cosine, sine)
};

struct LoweredBlock {
    std::vector<LoweredItem> items;
    int64_t members = 1;  // 1: the data are shared
    double cost = 0.0;    // complex multiply-adds per amplitude, `overhead` per operator included
};

// Lower a block whose operators have their positions and codes (whole: rotations as (cosine, sine)). False
// when it holds no rotation, or would hold more operators than before. `form`: its diagonals so far.
bool lower_block(const Plan& plan, const PassDesc& pd, const BlockDesc& blk, const std::vector<char>& moved,
                 int64_t batch, const Pool& pool, double overhead, bool whole, Choices& form, LoweredBlock* out);

}  // namespace lsg
