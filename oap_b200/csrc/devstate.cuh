// Device-resident state of a restart loop, read by the host once per restart.
#pragma once

#include "common.cuh"

namespace oapb {

struct DevState {
  double fnorm2;    // ||f||^2 of the current residual vector
  double hnorm2;
  int dgks;         // second Gram-Schmidt pass needed for the current column
  int converged;
  int status;       // bit 0: breakdown (||f|| = 0), bit 1: Schur sweep limit, bit 2: ||f|| not finite
  int dgks_count;
  int brk;          // the current basis vector replaces a zero residual (H[j][j-1] = 0)
  int brk_count;
  double scale;     // max |theta| over the wanted set
  double maxest;    // max relative Ritz estimate of the wanted set
  cplx beta_hat;    // H[k][k-1] after the shifts
  cplx sigma;       // Q[m-1][k-1]
  int symtri;       // eigensolves that took the Hermitian path
  int keep;         // vectors the last restart keeps (the next cycle's first step)
  int spike;        // row `keep` of H holds the kept Ritz vectors' coupling to the next basis vector
  int nosym;        // the basis lost the symmetry: the general path from here on
};

}  // namespace oapb
