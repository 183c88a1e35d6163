// One restart cycle of the plain FP64 Arnoldi loop on a dense operator in a
// single cooperative launch (cycle.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "devstate.cuh"

namespace oapb {

struct CycleArgs {
  const double* are;  // n x n row-major planes
  const double* aim;  // null for a real operator
  double* vre;        // basis, vector i at i n
  double* vim;
  double* fre;        // residual vector
  double* fim;
  cplx* H;            // m x m column-major
  const cplx* Q;      // restart rotations of the last small eigensolve (m x m)
  cplx* part;         // (m + 1) x ctas projection partials
  double* fpart;      // ctas norm partials
  unsigned* bar;      // grid barrier counter, zero at the launch
  DevState* st;
  int n, m;
  int j0;             // first step
  int restart;        // 1: V <- V Q[:, :j0], f <- (V Q)_j0 beta_hat + f sigma first
  double rho;
  uint64_t seed;      // breakdown vectors: seed + j
};

// The launch shape for (n, m): CTAs, rows per CTA, dynamic shared memory and
// whether each CTA's operator rows stay in shared memory for the cycle.
struct CyclePlan {
  int ctas = 0, rows = 0, segs = 1;
  bool resident = false;
  size_t smem = 0;
  int limit = 0;  // the device's shared memory per CTA
  int sms = 0;    // and its SMs
};

// false where the per-step kernels run instead: x, the basis rows and the
// work vectors of a CTA do not fit its shared memory, or m > 128
bool cycle_plan(int n, int m, bool cplx, CyclePlan* p);
// steps j0 .. m - 1 (st: fnorm2, hnorm2, dgks / breakdown counts, status)
int launch_cycle(const CyclePlan& p, const CycleArgs& a, cudaStream_t s);

}  // namespace oapb
