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

// The DGKS threshold of step j.  A step without the second pass multiplies what
// the basis has lost of its orthogonality by up to ||h|| / ||f||.  After a
// restart that keeps Ritz vectors (`spike`) the first two new vectors are formed
// against all of them; what they lack grows through the cycle and comes back
// with the kept vectors.  They take the second pass wherever it would grow at
// all (threshold 1).  With rho = 1 / 3.14 alone, 1024 evenly spaced values
// (m = 24 to 40, 6 to 12 wanted) left vectors 1e-2 from orthogonal, values 3700
// eps off or no convergence at all; now 45 eps and 1e-13.  (A threshold of 0.71
// was not enough.)  It costs one pass per restart: n = 2048, m = 24, 27 restarts
// 8.66 -> 8.91 ms.
__host__ __device__ inline double dgks_rho(double rho, bool spike, int keep, int j) {
  return spike && j >= keep && j < keep + 2 && rho < 1.0 ? 1.0 : rho;
}

}  // namespace oapb
