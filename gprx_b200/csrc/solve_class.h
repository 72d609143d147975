// solve_class.h — which way a triangular solve goes (tri_solve.cu): fixed by the whole
// solve, and with it the bits of a column.
#pragma once

namespace gprx {

// FEW: one cluster launch; MID, WIDE: recursion down to launches of 512 and of 256
// rows; BULK: down to products with the 128-row blocks' inverses.
enum SolveClass : int { SOLVE_FEW = 0, SOLVE_MID = 1, SOLVE_WIDE = 2, SOLVE_BULK = 3 };

// Of q right-hand sides with n rows, on the current device.
SolveClass solve_class(long long n, long long q);

}  // namespace gprx
