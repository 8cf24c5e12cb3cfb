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

}  // namespace eqg
