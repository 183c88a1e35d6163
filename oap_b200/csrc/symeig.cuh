// The restart loop's small eigensolve for a Hermitian (or real symmetric)
// operator, on a whole CTA.
//
// The Arnoldi matrix H of a Hermitian operator is real symmetric to rounding
// (its subdiagonal holds norms, its restart rows real numbers), whatever its
// sparsity.  Its eigen-decomposition is a parallel cyclic Jacobi iteration:
// m / 2 disjoint rotations per round (round-robin pairs), formed by m / 2
// threads and applied by all of them as 2 x 2 blocks J_i^T B J_k, so the
// depth of a sweep is m - 1 rounds instead of the m^2 / 2 dependent rotations
// of a tridiagonal QR sweep; six to nine sweeps converge.  The one-warp
// implicit QR it replaces spent about 650 cycles on each of its dependent
// rotations.  A cycle's check and restart at m = 24 took 299 us; the symmetric
// n = 2048 solve with 8 of 24 values at the spectrum's edge went from 27.8 to
// 11.0 ms with this solve and the restart below (fewer applications too).
//
// The restart keeps the Ritz vectors themselves (Wu and Simon's thick restart
// of the Lanczos method, mathematically the exact-shift restart): V <- V Q
// with Q the first `keep` eigenvectors, f unchanged, H = diag(theta) with the
// row beta e_m^T Q below it, so no shift sweeps follow.
//
// A matrix that carries such a row but has lost its symmetry (the basis's
// orthogonality went) cannot continue either way: the loop then starts again
// from the sum of the wanted Ritz vectors and keeps to the general path
// (DevState::nosym).
#pragma once

#include "hess.cuh"

namespace oapb {

constexpr int kSymMaxThreads = 512;
constexpr int kSymSweeps = 30;

// scratch of sym_eig besides A and Z (m x hess_ld(m) doubles each)
struct SymScratch {
  double* cs;   // 2 x (m / 2 + 1)
  double* key;  // m
  double* red;  // 16
  int* ord;     // m
  int* flag;    // 4
};
__host__ __device__ inline size_t sym_scratch_bytes(int m) {
  return sizeof(double) * (2 * (size_t)(m / 2 + 1) + m + 16) + sizeof(int) * ((size_t)m + 4);
}
__device__ __forceinline__ SymScratch sym_scratch(void* base, int m) {
  SymScratch s;
  s.cs = (double*)base;
  s.key = s.cs + 2 * (m / 2 + 1);
  s.red = s.key + m;
  s.ord = (int*)(s.red + 16);
  s.flag = s.ord + m;
  return s;
}

// pair i of round r of the round robin over M (even) indices: index 0 stays,
// the others rotate
__device__ __forceinline__ void sym_pair(int i, int r, int M, int& p, int& q) {
  const int N = M - 1;
  int a = i + r - 1, b = M - 2 - i + r;
  a = a >= N ? a - N : a;
  b = b >= N ? b - N : b;
  p = i == 0 ? 0 : 1 + a;
  q = 1 + b;
}

// Eigen-decomposition of the symmetric A (m x m, leading dimension ld,
// largest entry in [1, 2)): A becomes diagonal, Z (the identity on entry) the
// eigenvectors.  All nthr threads of the CTA.
static __device__ bool cta_jacobi(double* A, double* Z, int m, int ld, const SymScratch& S, int tid, int nthr) {
  const int M = (m + 1) & ~1, h = M / 2;
  for (int sweep = 0; sweep < kSymSweeps; ++sweep) {
    if (tid == 0) S.flag[0] = 0;
    for (int r = 0; r < M - 1; ++r) {
      __syncthreads();
      if (tid < h) {
        int p, q;
        sym_pair(tid, r, M, p, q);
        double c = 1, s = 0;
        if (p < m && q < m) {
          const double app = A[p + p * ld], aqq = A[q + q * ld], apq = A[p + q * ld];
          // negligible beside its diagonal entries, or a tenth of an ulp of the largest entry
          if (!(fabs(apq) <= 1.1e-16 * (fabs(app) + fabs(aqq)) || fabs(apq) <= 2e-17)) {
            // tan 2t = 2 apq / (aqq - app): cos 2t = |d| / r, the small angle
            const double d = aqq - app, g = 2 * apq;
            const double ir = rsqrt(fma(d, d, g * g));
            const double c2 = fma(0.5 * fabs(d), ir, 0.5);
            const double rc = rsqrt(c2);
            c = c2 * rc;
            s = (d >= 0 ? 0.5 : -0.5) * g * ir * rc;
            S.flag[0] = 1;
          }
        }
        S.cs[2 * tid] = c;
        S.cs[2 * tid + 1] = s;
      }
      __syncthreads();
      // B <- J_i^T B J_k on every 2 x 2 block, J = [c s; -s c]
      for (int e = tid; e < h * h; e += nthr) {
        const int i = e % h, k = e / h;
        int p, q, u, v;
        sym_pair(i, r, M, p, q);
        sym_pair(k, r, M, u, v);
        const double ci = S.cs[2 * i], si = S.cs[2 * i + 1], ck = S.cs[2 * k], sk = S.cs[2 * k + 1];
        const bool in_q = q < m && p < m, in_v = v < m && u < m;
        if (!in_q || !in_v) {  // the padding index of an odd m: c = 1, s = 0 for its pair
          if (!in_q && !in_v) continue;
          if (!in_q) {  // one row (p or q, whichever is real), columns u, v
            const int x = p < m ? p : q;
            const double b0 = A[x + u * ld], b1 = A[x + v * ld];
            A[x + u * ld] = ck * b0 - sk * b1;
            A[x + v * ld] = sk * b0 + ck * b1;
          } else {
            const int x = u < m ? u : v;
            const double b0 = A[p + x * ld], b1 = A[q + x * ld];
            A[p + x * ld] = ci * b0 - si * b1;
            A[q + x * ld] = si * b0 + ci * b1;
          }
          continue;
        }
        const double b00 = A[p + u * ld], b01 = A[p + v * ld], b10 = A[q + u * ld], b11 = A[q + v * ld];
        const double t00 = ci * b00 - si * b10, t01 = ci * b01 - si * b11;
        const double t10 = si * b00 + ci * b10, t11 = si * b01 + ci * b11;
        double n01 = sk * t00 + ck * t01, n10 = ck * t10 - sk * t11;
        if (i == k && si != 0) n01 = n10 = 0;
        A[p + u * ld] = ck * t00 - sk * t01;
        A[p + v * ld] = n01;
        A[q + u * ld] = n10;
        A[q + v * ld] = sk * t10 + ck * t11;
      }
      for (int e = tid; e < h * m; e += nthr) {
        const int x = e % m, k = e / m;
        int u, v;
        sym_pair(k, r, M, u, v);
        if (u >= m || v >= m) continue;
        const double ck = S.cs[2 * k], sk = S.cs[2 * k + 1];
        const double z0 = Z[x + u * ld], z1 = Z[x + v * ld];
        Z[x + u * ld] = ck * z0 - sk * z1;
        Z[x + v * ld] = sk * z0 + ck * z1;
      }
    }
    __syncthreads();
    const int more = S.flag[0];
    __syncthreads();
    if (!more) return true;
  }
  return false;
}

// The check and restart of hess_core for a real symmetric H (arguments and
// outputs as there; a.keep_sym vectors are kept).  All nthr threads of the
// CTA; returns false (nothing written) when H is not symmetric to a tenth of
// the residual goal: hess_core then takes it.
static __device__ bool sym_eig(const HessArgs& a, double* A, double* Z, const SymScratch& S, int tid, int nthr) {
  const int m = a.m, k = a.k, ld = hess_ld(m), mm = m * m;
  const int warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
  DevState* st = a.st;
  const int nosym = st->nosym;
  const double beta = sqrt(st->fnorm2);
  double mx = 0;
  for (int e = tid; e < mm; e += nthr) mx = fmax(mx, fmax(fabs(a.Hin[e].re), fabs(a.Hin[e].im)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) S.red[warp] = mx;
  __syncthreads();
  for (int w = 0; w < nw; ++w) mx = fmax(mx, S.red[w]);
  int ex = 0;
  if (mx > 0 && mx <= 1.7e308) frexp(mx, &ex);
  ex = ex > 1000 ? 1000 : (ex < -1000 ? -1000 : ex);
  const double sig = ldexp(1.0, 1 - ex), isig = ldexp(1.0, ex - 1), rtol = 0.1 * a.tol;
  int bad = 0, row = 0;
  for (int e = tid; e < mm; e += nthr) {
    const int r = e % m, c = e / m;
    const cplx x = a.Hin[e], y = a.Hin[c + r * m];
    const double xr = sig * x.re, yr = sig * y.re;
    if (!(fabs(xr - yr) <= rtol && fabs(sig * x.im) <= rtol)) bad = 1;
    if (r > c + 1 && (x.re != 0 || x.im != 0)) row = 1;
    A[r + c * ld] = 0.5 * (xr + yr);
    Z[r + c * ld] = r == c ? 1.0 : 0.0;
  }
  bad = __syncthreads_or(bad || nosym || !(a.tol > 0));
  row = __syncthreads_or(row);
  if (bad && !row) return false;
  if (!cta_jacobi(A, Z, m, ld, S, tid, nthr)) {
    if (tid == 0) {
      st->status |= 2;
      st->converged = 0;
    }
    return true;
  }
  for (int i = tid; i < m; i += nthr) {
    const double kv = sort_key(cplx{A[i + i * ld], 0}, a.which);
    S.key[i] = (kv != kv) ? INFINITY : kv;
  }
  __syncthreads();
  for (int i = tid; i < m; i += nthr) {
    int r = 0;
    for (int j = 0; j < m; ++j) r += (S.key[j] < S.key[i]) || (S.key[j] == S.key[i] && j < i);
    S.ord[r] = i;
  }
  __syncthreads();
  double scale = 0, maxest = 0;
  for (int q = 0; q < k; ++q) {
    scale = fmax(scale, fabs(A[S.ord[q] + S.ord[q] * ld]));
    maxest = fmax(maxest, fabs(Z[m - 1 + S.ord[q] * ld]));
  }
  scale *= isig;
  if (scale == 0) scale = 1;
  maxest *= beta / scale;
  const int nvec = a.nvec > k ? (a.nvec < m ? a.nvec : m) : k;
  for (int q = tid; q < m; q += nthr) {
    const int o = S.ord[q];
    a.order[q] = o;
    a.ritz[q] = cplx{isig * A[o + o * ld], 0};
    if (q < nvec) a.est[q] = beta * fabs(Z[m - 1 + o * ld]) / scale;
  }
  for (int e = tid; e < m * nvec; e += nthr) a.Y[e] = cplx{Z[e % m + S.ord[e / m] * ld], 0};
  const int conv = !bad && maxest <= a.tol;
  const int go = !conv && a.do_shift;
  const int keep = bad ? 0 : a.keep_sym;
  if (tid == 0) {
    st->converged = conv;
    st->scale = scale;
    st->maxest = maxest;
    if (!bad) st->symtri += 1;
    if (go) {
      st->keep = keep;
      st->spike = !bad;
      st->nosym = bad;
      st->beta_hat = cplx{bad ? 1.0 : 0.0, 0};
      st->sigma = cplx{bad ? 0.0 : 1.0, 0};
    }
  }
  if (!go) return true;
  // (Hin, which Hout may alias, was last read before the barriers above)
  for (int e = tid; e < mm; e += nthr) {
    const int r = e % m, c = e / m;
    double h = 0, z = 0;
    if (c < keep) {
      const int o = S.ord[c];
      z = Z[r + o * ld];
      if (r == c) h = isig * A[o + o * ld];
      if (r == keep) h = beta * Z[m - 1 + o * ld];
    } else if (bad && c == 0) {
      for (int q = 0; q < k; ++q) z += Z[r + S.ord[q] * ld];
    }
    a.Hout[e] = cplx{h, 0};
    a.Qout[e] = cplx{z, 0};
  }
  return true;
}

// dynamic shared memory of k_symeig
__host__ __device__ inline size_t sym_smem_bytes(int m) {
  return sizeof(double) * 2 * (size_t)hess_ld(m) * m + sym_scratch_bytes(m);
}
inline int sym_threads(int m) { return m <= 16 ? 64 : m <= 24 ? 160 : m <= 40 ? 256 : kSymMaxThreads; }

// *delivered = 1 when the symmetric path took the matrix (k_hess follows with
// skip = delivered)
static __global__ void __launch_bounds__(kSymMaxThreads) k_symeig(HessArgs a, int* delivered) {
  extern __shared__ __align__(16) unsigned char sym_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  double* A = reinterpret_cast<double*>(sym_dyn);
  double* Z = A + (size_t)hess_ld(a.m) * a.m;
  const bool got = sym_eig(a, A, Z, sym_scratch(Z + (size_t)hess_ld(a.m) * a.m, a.m), threadIdx.x, blockDim.x);
  if (threadIdx.x == 0) *delivered = got;
}

}  // namespace oapb
