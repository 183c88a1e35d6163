// The restart loop's small eigensolve for a Hermitian (or real symmetric)
// operator, on a whole CTA.
//
// The Arnoldi matrix H of a Hermitian operator is real symmetric to rounding
// (its subdiagonal holds norms, its restart rows real numbers), whatever its
// sparsity.  Its eigen-decomposition is a parallel cyclic Jacobi iteration:
// m / 2 disjoint rotations per round (round-robin pairs), applied by all
// threads as 2 x 2 blocks J_i^T B J_k, so the depth of a sweep is m - 1 rounds
// instead of the dependent rotations of tridiagonal QR sweeps; six or seven
// sweeps converge at m <= 32, nine or ten at m = 96.  The one-warp
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

// A and Z are padded to an even number of rows (the pad's entries are zero,
// so its pairs never rotate)
__host__ __device__ __forceinline__ int sym_even(int m) { return (m + 1) & ~1; }
__host__ __device__ __forceinline__ int sym_ld(int m) { return sym_even(m) + 1; }
__host__ __device__ inline size_t sym_matrix(int m) { return (size_t)sym_ld(m) * sym_even(m); }

// scratch of sym_eig besides A and Z (sym_matrix(m) doubles each)
struct SymScratch {
  double* cs;   // two rounds' rotations: 2 x 2 x (m / 2 + 1)
  double* key;  // m
  double* red;  // 16
  int* ord;     // m
  int* flag;    // 4
};
__host__ __device__ inline size_t sym_scratch_bytes(int m) {
  return sizeof(double) * (4 * (size_t)(m / 2 + 1) + m + 16) + sizeof(int) * ((size_t)m + 4);
}
__device__ __forceinline__ SymScratch sym_scratch(void* base, int m) {
  SymScratch s;
  s.cs = (double*)base;
  s.key = s.cs + 4 * (m / 2 + 1);
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

// FP64 <-> FP32 of values in FP32's normal range (smaller ones become zero) on
// the integer pipe: the conversion instructions' latency sits on a round's
// critical path
__device__ __forceinline__ float sym_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mag = ((hi & 0x7fffffffu) - (896u << 20)) << 3 | lo >> 29;
  return (hi & 0x7fffffffu) >= (897u << 20) ? __uint_as_float((hi & 0x80000000u) | mag) : 0.f;
}
__device__ __forceinline__ double sym_f64(float x) {
  const unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
  if (mag < 0x00800000u) return 0.0;
  return __hiloint2double((int)((b & 0x80000000u) | ((mag >> 3) + (896u << 20))), (int)(b << 29));
}

// The rotation J = [c s; -s c] that annihilates apq (J^T B J), the identity
// where apq is negligible beside its diagonal entries or a tenth of an ulp of
// the largest entry (which is in [1, 2)).  The angle comes from FP32: its
// error leaves about 1e-7 of apq, less than the next sweep removes.  c is one
// Halley step (cubic, 1e-7 -> 1e-21) from the FP32 reciprocal square root, so
// the rotation is orthonormal to FP64 rounding.  Returns whether the angle is
// above 1e-8: what smaller ones leave off the diagonal is of second order,
// below rounding.
__device__ __forceinline__ bool sym_rotation(double app, double aqq, double apq, double& c, double& s) {
  c = 1;
  s = 0;
  if (fabs(apq) <= 1.1e-16 * (fabs(app) + fabs(aqq)) || fabs(apq) <= 2e-17) return false;
  // tan 2t = 2 apq / (aqq - app), |t| <= pi / 4
  const float d = sym_f32(aqq - app), g = 2.f * sym_f32(apq), w = fmaf(d, d, g * g);
  const float t = __fdividef(copysignf(1.f, d) * g, fabsf(d) + w * rsqrtf(w));
  const double td = sym_f64(t), x1 = fma(td, td, 1.0), y = sym_f64(rsqrtf(fmaf(t, t, 1.f)));
  const double e = fma(-x1, y * y, 1.0), p = fma(0.375, e, 0.5);
  c = fma(y * e, p, y);
  s = fma(td * y * e, p, td * y);
  return !(fabsf(t) <= 1e-8f);
}

// B <- J_i^T B J_k for the 2 x 2 block of rows p, q and columns u, v
__device__ __forceinline__ void sym_block(double* A, int ld, int p, int q, int u, int v, double ci, double si, double ck,
                                          double sk) {
  const double b00 = A[p + u * ld], b01 = A[p + v * ld], b10 = A[q + u * ld], b11 = A[q + v * ld];
  const double t00 = ci * b00 - si * b10, t01 = ci * b01 - si * b11;
  const double t10 = si * b00 + ci * b10, t11 = si * b01 + ci * b11;
  A[p + u * ld] = ck * t00 - sk * t01;
  A[p + v * ld] = sk * t00 + ck * t01;
  A[q + u * ld] = ck * t10 - sk * t11;
  A[q + v * ld] = sk * t10 + ck * t11;
}

// Z <- Z J on the pairs k0, k0 + dk, ... of round r, rows x0, x0 + 32, ...
__device__ __forceinline__ void sym_z(double* Z, int m, int ld, int M, int r, const double* cs, int k0, int dk, int x0) {
  for (int k = k0; k < M / 2; k += dk) {
    int u, v;
    sym_pair(k, r, M, u, v);
    const double ck = cs[2 * k], sk = cs[2 * k + 1];
    if (sk == 0) continue;
    for (int x = x0; x < m; x += 32) {
      const double z0 = Z[x + u * ld], z1 = Z[x + v * ld];
      Z[x + u * ld] = ck * z0 - sk * z1;
      Z[x + v * ld] = sk * z0 + ck * z1;
    }
  }
}

// Eigen-decomposition of the symmetric A (m x m padded, leading dimension ld,
// largest entry in [1, 2)): A becomes diagonal, Z (the identity on entry) the
// eigenvectors; false when the sweeps ran out.  All nthr threads of the CTA.
//
// A round's time is latency: one rotation's arithmetic, the block update and
// two barriers (k_symeig, m = 24: 154 us with an FP64 rotation and A and Z on the
// same threads, 90 us here; m = 32: 237 and 144 us).  For m <= 32 on 512 threads
// one half updates A and the other Z.  Tried and not kept: every thread forming
// the two rotations of its block itself, with one barrier per round and two copies
// of A (a seventh slower at m = 24, a fifth at m = 32: the repeated FP64
// arithmetic).
static __device__ bool cta_jacobi(double* A, double* Z, int m, int ld, const SymScratch& S, int tid, int nthr) {
  const int M = sym_even(m), h = M / 2;
  const bool split = h <= 16 && nthr >= 512;
  const bool on_a = !split || tid < 256, on_z = !split || tid >= 256;
  const int sh = h <= 16 ? 4 : 5;
  const int i0 = tid & ((1 << sh) - 1), k0 = tid >> sh, dk = (split ? 256 : nthr) >> sh;
  const int tz = split ? tid - 256 : tid, zk0 = tz >> 5, zdk = (split ? nthr - 256 : nthr) >> 5, zx0 = tz & 31;
  for (int sweep = 0; sweep < kSymSweeps; ++sweep) {
    if (tid == 0) S.flag[0] = 0;
    for (int r = 0; r < M - 1; ++r) {
      double* cs = S.cs + (r & 1) * 2 * h;
      __syncthreads();
      if (tid < h) {
        int p, q;
        sym_pair(tid, r, M, p, q);
        if (sym_rotation(A[p + p * ld], A[q + q * ld], A[p + q * ld], cs[2 * tid], cs[2 * tid + 1])) S.flag[0] = 1;
      }
      __syncthreads();
      if (on_a)
        for (int i = i0; i < h; i += 1 << sh) {
          int p, q;
          sym_pair(i, r, M, p, q);
          const double ci = cs[2 * i], si = cs[2 * i + 1];
          for (int k = k0; k < h; k += dk) {
            int u, v;
            sym_pair(k, r, M, u, v);
            sym_block(A, ld, p, q, u, v, ci, si, cs[2 * k], cs[2 * k + 1]);
          }
        }
      if (on_z) sym_z(Z, m, ld, M, r, cs, zk0, zdk, zx0);
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
  const int m = a.m, k = a.k, ld = sym_ld(m), mm = m * m;
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
  if (m & 1)  // the pad
    for (int e = tid; e <= m; e += nthr) {
      A[m + e * ld] = A[e + m * ld] = 0;
      Z[m + e * ld] = Z[e + m * ld] = 0;
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
    // (the imaginary parts all tie: the largest |value| first, which a restarted
    // space finds; in diagonal order the wanted set was an arbitrary one inside
    // the spectrum, another after every restart, and the loop did not converge)
    const bool ties = a.which == OAPB_SORT_LARGEST_IM || a.which == OAPB_SORT_SMALLEST_IM;
    const double kv = ties ? -fabs(A[i + i * ld]) : sort_key(cplx{A[i + i * ld], 0}, a.which);
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
  return sizeof(double) * 2 * sym_matrix(m) + sym_scratch_bytes(m);
}

// *delivered = 1 when the symmetric path took the matrix (k_hess follows with
// skip = delivered)
static __global__ void __launch_bounds__(kSymMaxThreads) k_symeig(HessArgs a, int* delivered) {
  extern __shared__ __align__(16) unsigned char sym_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  double* A = reinterpret_cast<double*>(sym_dyn);
  double* Z = A + sym_matrix(a.m);
  const bool got = sym_eig(a, A, Z, sym_scratch(Z + sym_matrix(a.m), a.m), threadIdx.x, blockDim.x);
  if (threadIdx.x == 0) *delivered = got;
}

}  // namespace oapb
