// Which systems the kernels' 32-bit offsets take, as plain host arithmetic
// (no CUDA: also compiled by the tests).
#pragma once

#include <climits>
#include <cstdint>

namespace eqg {

// Systems of `cells` cells with nd neighbours each and blocks of bb values
// that the two-colour form takes: those whose diagonal and off-diagonal blocks
// have 32-bit value offsets, as the general form requires of the blocks that it
// stores.  Larger ones are left to the general form, which stores fewer blocks
// where the pattern has fewer and refuses what it cannot number.  (The
// two-colour kernels number rows in 32 bits and values in 64.)
inline bool two_colour_fits(int64_t cells, int nd, int bb) { return (double)cells * (nd + 1) * bb < (double)INT_MAX; }

// Products M J that get a position plan (spgemm_plan_kernel): 8 bytes for each
// contribution, of which the operators of a grid make at most six per entry of
// J (a cell's faces) or one per entry of the product, so that their number
// stays below 2^31, and 4 bytes for each entry of the product (20 while it is
// built).  Larger Jacobians are merged row by row, which needs no memory.
constexpr int64_t kPlanOperand = (1 << 27) - 1;
inline bool plan_fits(int64_t operand_nnz, int64_t product_nnz)
{
    return operand_nnz <= kPlanOperand && product_nnz < (int64_t)INT_MAX / 2;
}

}  // namespace eqg
