// Small dense kernels of the restart loop and of the block methods' checks,
// FP64 complex (FP32 working arithmetic in k_hess_f32).
//
// k_hess works on the m x m upper Hessenberg H of the Arnoldi factorization
// (column-major, m <= kMaxM):
//   1. complex Schur form T = Z^H H Z by single-shift QR sweeps (Givens
//      bulge chasing, Wilkinson shifts, deflation at
//      |T[i][i-1]| <= eps (|T[i-1][i-1]| + |T[i][i]|)), the restatement of
//      calculateTriangularHEigens (ArnoldiProcedures.cpp:341-349) with a
//      shifted, deflating iteration instead of the reference's unshifted
//      one; for a Hermitian H (a Hermitian or real symmetric operator) beyond
//      the sizes of symeig.cuh the implicit symmetric tridiagonal QR instead;
//   2. Ritz values = diag(T), sorted by the ArnUtils order
//      (ArnoldiUtils.cpp:24-50); wanted = first k (getWanted,
//      ArnoldiProcedures.cpp:381-398);
//   3. eigenvectors y_q = Z u_q of the wanted values (back substitution on
//      T) and Ritz estimates beta |e_m^T y_q|;
//   4. if not converged: exact shifts with the values after the first `keep`
//      (iram_shiftedQRIterations, oapGenericArnoldiApi.h:186-222) on H,
//      Q accumulating the rotations, H compressed to its leading keep x keep
//      block.
// With `dense` set the input is a general matrix, first reduced to
// Hessenberg form by Householder reflectors accumulated into Z.  The input
// is scaled by a power of two (exact) so that the rotations need no
// overflow branches.
//
// Work layout: T and Z are column-major with an odd leading dimension
// hess_ld(m), so a lane-per-column access (row rotations) and a
// lane-per-row access (column rotations) are both free of bank conflicts.
// A QR sweep runs its chain of rotations on one warp, in registers (the 2 x 2
// window and the bulge, one shuffle per rotation) while the lanes apply each
// row rotation to their columns; the column rotations of the sweep, and those
// on Z, are applied after the chain (each lane the whole sequence to its row),
// those on Z by another warp beside the next sweep.  The eigenvector back
// substitutions run one lane per eigenvector (T read by broadcast).  For m <= 32
// the kernel's four warps share the Householder reduction and the product
// Y = Z U.
//
// Every loop is bounded (30 m sweeps for the Schur form); hitting the bound
// sets bit 1 of DevState::status and the kernel returns.
#pragma once

#include "common.cuh"
#include "devstate.cuh"

namespace oapb {

constexpr int kMaxM = 256;

struct HessArgs {
  const cplx* Hin;  // m x m column-major input
  cplx* Hout;       // compressed H after the shifts (may alias Hin)
  cplx* Qout;       // accumulated shift rotations (m x m)
  cplx* ritz;       // m Ritz values in sort order
  cplx* Y;          // k eigenvectors of H (column q at Y + q m)
  double* est;      // k relative Ritz estimates
  int* order;       // m sort order (indices into diag(T))
  DevState* st;
  cplx* gws;        // global workspace (hess_ws_cplx(m)) when shared memory is too small
  int m, k, nvec, which, do_shift, real_shifts, dense, use_beta;
  int keep = 0;      // vectors a restart keeps (k <= keep < m): general path,
  int keep_sym = 0;  // symmetric path
  double tol;
  double beta;      // used when use_beta == 0 (dense mode: residual norms come separately)
  const int* skip = nullptr;  // k_hess: when set and *skip != 0, return at once (another solver delivered)
};

// Vectors a restart keeps on the symmetric path: one guard vector beyond the
// wanted.  It takes most of what more would give (over 32 operators with 8 of
// 24 at a spectrum's edge, 7800 applications with none, 5600 with one, 4600
// with five; more of them also leave a warm start little to save).  In a space
// of fewer than k + 4 vectors it takes too much of what a restart adds (24 Gaussian
// symmetric operators of 80 to 150 rows, one wanted: m = k + 2 4017 restarts in
// all without it and 7266 with it, k + 3 1892 and 1982, k + 4 1116 and 971, k + 5
// 752 and 594).  On the general path a restart costs as much as 10 - 30
// applications (its Schur form), and more kept vectors mean more restarts: the
// wanted alone.
__host__ __device__ inline int restart_keep(int m, int k, bool sym) { return sym && m - k >= 4 ? k + 1 : k; }

// leading dimension of the T / Z work arrays (odd)
__host__ __device__ __forceinline__ int hess_ld(int m) { return m | 1; }
// scratch (rotation list and eigenvector columns), in cplx
__host__ __device__ __forceinline__ size_t hess_scratch_cplx(int m) { return (size_t)m * 32 + 2 * (size_t)m + 2; }
// whole k_hess workspace: T, Z and the scratch
__host__ __device__ __forceinline__ size_t hess_ws_cplx(int m) {
  return 2 * (size_t)hess_ld(m) * m + hess_scratch_cplx(m);
}

// precision constants of the working type
template <typename R>
struct HessK;
template <>
struct HessK<double> {
  static constexpr double eps = 2.220446049250313e-16, tiny = 1e-300, big = 1e150, unbig = 1e-150;
  static constexpr double tiny2 = 1e-280;  // |x|^2 + |y|^2 of a negligible pair (prescaled matrix)
};
template <>
struct HessK<float> {
  static constexpr float eps = 1.1920929e-7f, tiny = 1e-37f, big = 1e15f, unbig = 1e-15f;  // big^2 stays finite
  static constexpr float tiny2 = 1e-36f;
};

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float rsqrt_t(float a) { return rsqrtf(a); }
__device__ __forceinline__ double rsqrt_t(double a) { return rsqrt(a); }
__device__ __forceinline__ float sqrt_t(float a) { return sqrtf(a); }
__device__ __forceinline__ float abs_t(float a) { return fabsf(a); }
__device__ __forceinline__ double abs_t(double a) { return fabs(a); }
__device__ __forceinline__ double sqrt_t(double a) { return sqrt(a); }

// a b + c with fused multiply-adds
template <typename Cx>
__device__ __forceinline__ Cx cfma(Cx a, Cx b, Cx c) {
  return {fma_t(a.re, b.re, fma_t(-a.im, b.im, c.re)), fma_t(a.re, b.im, fma_t(a.im, b.re, c.im))};
}
// a b + c d
template <typename Cx>
__device__ __forceinline__ Cx cfma2(Cx a, Cx b, Cx c, Cx d) {
  return cfma(a, b, c * d);
}

// p, known to lie in shared memory: its accesses then need no generic address
template <typename P>
__device__ __forceinline__ P* as_shared(P* p) {
  return static_cast<P*>(__cvta_shared_to_generic(__cvta_generic_to_shared(p)));
}

// one complex entry in one access (T, Z and the rotation lists start on 16
// bytes; the structs alone promise only a component's alignment)
__device__ __forceinline__ cplx cload(const cplx* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ cplxf cload(const cplxf* p) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void cstore(cplx* p, cplx v) { *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im); }
__device__ __forceinline__ void cstore(cplxf* p, cplxf v) { *reinterpret_cast<float2*>(p) = make_float2(v.re, v.im); }

// principal square root of z (prescaled entries: |z| stays far inside the
// range), re >= 0
template <typename Cx>
__device__ __forceinline__ Cx csqrt_s(Cx z) {
  using R = decltype(Cx::re);
  const R r = sqrt_t(abs2(z));
  const R u = R(0.5) * (r + abs_t(z.re));
  const R iu = rsqrt_t(u > 0 ? u : R(1));
  const R t = u > 0 ? u * iu : R(0), hh = u > 0 ? R(0.5) * z.im * iu : R(0);  // sqrt(u), im / (2 sqrt(u))
  return z.re >= 0 ? Cx{t, hh} : Cx{abs_t(hh), z.im >= 0 ? t : -t};
}

__device__ __forceinline__ double warp_sum_t(double v) { return warp_sum(v); }
__device__ __forceinline__ float warp_sum_t(float v) { return warp_sumf(v); }

#define TT_(i, j) T[(i) + (j) * ld]
#define ZZ_(i, j) Z[(i) + (j) * ld]

__device__ __forceinline__ double sort_key(cplx v, int which) {
  switch (which) {
    case 0: return -(v.re * v.re + v.im * v.im);
    case 1: return -v.re;
    case 2: return -v.im;
    case 3: return v.re * v.re + v.im * v.im;
    case 4: return v.re;
    default: return v.im;
  }
}

// |re| + |im| (LAPACK's CABS1): the deflation test only needs a norm-equivalent
__device__ __forceinline__ double cabs1(cplx a) { return fabs(a.re) + fabs(a.im); }
__device__ __forceinline__ float cabs1(cplxf a) { return fabsf(a.re) + fabsf(a.im); }

template <typename Cx>
__device__ __forceinline__ bool negligible(const Cx* T, int ld, int l) {
  using R = decltype(Cx::re);
  R s = cabs1(TT_(l - 1, l - 1)) + cabs1(TT_(l, l));
  if (s == 0) s = HessK<R>::tiny;
  return cabs1(TT_(l, l - 1)) <= HessK<R>::eps * s;
}

__device__ __forceinline__ cplx shfl_c(cplx v, int src) {
  return cplx{__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}
__device__ __forceinline__ cplxf shfl_c(cplxf v, int src) {
  return cplxf{__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
}

// The largest l in [1, h] with T[l][l-1] negligible, else 0 (all lanes).
template <typename Cx>
static __device__ int find_split(const Cx* T, int ld, int h, int lane) {
  for (int base = h; base >= 1; base -= 32) {
    const int l = base - lane;
    const bool f = l >= 1 && negligible(T, ld, l);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (bal) return base - (__ffs(bal) - 1);
  }
  return 0;
}

// One single-shift QR sweep on the active window [l, h] of Hessenberg T,
// applied to whole rows / columns of T (the final T is G T G^H with G =
// G_{h-1} ... G_l); Z <- Z G_l^H ... G_{h-1}^H.
// T must be prescaled (hess_core).
//
// warp_chain: the rotations (p, q at rot[2 k], rot[2 k + 1]) and their left
// products.  Rotation k needs the bulge pair left by rotation k - 1, so they
// form a dependent chain, which bounds the sweep.  It runs in registers:
// every lane carries the pair (x, y) = (T[k][k-1], T[k+1][k-1]) and the
// window D = T[k][k], F = T[k+1][k], G = T[k+1][k+1] (E = T[k][k+1] comes from
// the lane that owns column k + 1).  With r^2 = |x|^2 + |y|^2 and the
// unnormalised row N1 = x F - y D, N2 = x G - y E, the next pair's x is
// (N1 x + N2 y) / r^2 and the next D is (N2 conj(x) - N1 conj(y)) / r^2: both
// need only products that run beside the reciprocal square root, one
// multiplication after it.  A pair whose squares sum below tiny2 (far below
// the working precision relative to the matrix) gives the identity.
// Meanwhile lane c applies each row rotation to column c (its row-k entry
// carried in a register); rows k + 2 and on are read a step ahead.
//
// cols_rows: after the chain, one lane per row applies all column rotations to
// its row of T or Z.  Left and right rotations commute, so the result is
// G T G^H as in the interleaved sweep; the entries below the subdiagonal that
// the interleaved sweep never fills come out of this order at rounding level
// and are set to zero.  With several warps only the chain is serial: the next
// sweep starts when the rows of T are done, and the rows of Z go to another
// warp, which works beside it (two rotation lists in turn).
//
// Clocks per rotation at m = 32, FP64 (FP32): one warp, the window normalised
// before its products and the column rotations of T and Z after the chain, 457
// + 265 (323 + 211); now 334 + 112 (197 + 72), at m = 64 413 + 104 before 582 +
// 487.  A Schur form with 24 exact shifts, m = 32: 1097 -> 715 us (684 -> 392);
// m = 64, 56 shifts: 6.05 -> 3.00 ms (4.00 -> 1.67).  An FP64 instruction holds
// a warp's FP64 port for about 4 clocks: the chain's 80 are what bounds it.
// (Column rotations of T inside the chain's loop, a step behind it, made that
// 512 clocks per rotation.)
// NT: columns per lane (c = lane + 32 t, t < NT); m <= 32 NT.
template <typename Cx, int NT>
static __device__ __forceinline__ void warp_chain(Cx* T, int m, int ld, int l, int h, Cx mu, Cx* rot, int lane) {
  using R = decltype(Cx::re);
  const int nt = (m + 31) >> 5;
  const Cx zero = {0, 0};
  Cx carry[NT], b[NT], bn[NT];
  bool own[NT];
  const int r2nd = l + 2 < h ? l + 2 : h;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int c = lane + 32 * t;
    own[t] = t < nt && c >= l && c < m;
    carry[t] = own[t] ? cload(&TT_(l, c)) : zero;
    b[t] = own[t] ? cload(&TT_(l + 1, c)) : zero;
    bn[t] = own[t] ? cload(&TT_(r2nd, c)) : zero;
  }
  Cx D = cload(&TT_(l, l)), F = cload(&TT_(l + 1, l)), G = cload(&TT_(l + 1, l + 1));
  Cx s2 = cload(&TT_(r2nd, l + 1)), g2 = cload(&TT_(r2nd, r2nd));
  Cx x = D - mu, y = F;
  for (int k = l;; ++k) {
    // the step after the next one's inputs: row k + 3 (the last row instead
    // beyond the window, not used then)
    const int rn = k + 3 < h ? k + 3 : h, cn = rn - 1;
    Cx bnn[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) bnn[t] = own[t] ? cload(&TT_(rn, lane + 32 * t)) : zero;
    const Cx s3 = cload(&TT_(rn, cn)), g3 = cload(&TT_(rn, rn));
    // row k's entry of column k + 1
    const int c1 = k + 1;
    Cx e = carry[0];
#pragma unroll
    for (int t = 1; t < NT; ++t)
      if (t == (c1 >> 5)) e = carry[t];
    const Cx E = shfl_c(e, c1 & 31);
    const R r2 = fma_t(x.re, x.re, x.im * x.im) + fma_t(y.re, y.re, y.im * y.im);
    const Cx ny = -y;
    const Cx N1 = cfma2(ny, D, x, F), N2 = cfma2(ny, E, x, G);
    const Cx X = cfma2(N1, x, N2, y), Dn = cfma2(N2, conj(x), -N1, conj(y));
    const bool ok = r2 > HessK<R>::tiny2;
    const R ir = rsqrt_t(ok ? r2 : R(1));
    const R ir2 = ir * ir;
    const Cx p = ok ? Cx{x.re * ir, -x.im * ir} : Cx{1, 0};
    const Cx q = ok ? Cx{y.re * ir, -y.im * ir} : zero;
    cstore(rot + 2 * k, p);  // every lane stores the same values
    cstore(rot + 2 * k + 1, q);
    x = ok ? ir2 * X : F;
    D = ok ? ir2 * Dn : G;
    y = s2 * conj(q);  // T[k+2][k], the bulge
    F = s2 * p;        // T[k+2][k+1]
    G = g2;
    s2 = s3;
    g2 = g3;
    const Cx pc = conj(p), nqc = -conj(q);
    // row rotation k on the lanes' columns (rows k, k + 1)
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const Cx top = cfma2(p, carry[t], q, b[t]);
      carry[t] = cfma2(nqc, carry[t], pc, b[t]);
      if (own[t]) cstore(&TT_(k, lane + 32 * t), top);
      b[t] = bn[t];
      bn[t] = bnn[t];
    }
    if (k + 1 >= h) break;
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
    if (own[t]) cstore(&TT_(h, lane + 32 * t), carry[t]);
}

// U column rotations from k0 on, on one row (t: its entry of column 0; c: its
// entry of column k0, then of k0 + U); all are read before the first is stored
template <typename Cx, bool WT, int U>
static __device__ __forceinline__ void cols_block(Cx* t, int ld, int i, int k0, const Cx* rot, Cx& c) {
  const Cx zero = {0, 0};
  Cx p[U], q[U], nb[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    p[u] = cload(rot + 2 * (k0 + u));
    q[u] = cload(rot + 2 * (k0 + u) + 1);
    nb[u] = cload(t + (k0 + u + 1) * ld);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const Cx v = cfma2(c, conj(p[u]), nb[u], conj(q[u]));
    cstore(t + (k0 + u) * ld, WT && k0 + u + 2 <= i ? zero : v);
    c = cfma2(-c, q[u], nb[u], p[u]);
  }
}

// column rotations l .. h-1 on row i of T (WT, i <= h; the entries below the
// window's subdiagonal, rows i >= k + 2 of column k, are set to zero, and rows
// below h hold zeros in these columns) or of Z
template <typename Cx, bool WT>
static __device__ __forceinline__ void cols_rows(Cx* M, int ld, int i, int l, int h, const Cx* rot) {
  Cx* t = M + i;
  Cx c = cload(t + l * ld);
  int k = l;
  for (; k + 4 <= h; k += 4) cols_block<Cx, WT, 4>(t, ld, i, k, rot, c);
  if (k + 2 <= h) {
    cols_block<Cx, WT, 2>(t, ld, i, k, rot, c);
    k += 2;
  }
  if (k < h) cols_block<Cx, WT, 1>(t, ld, i, k, rot, c);
  cstore(t + h * ld, c);
}

// barriers of the NW warps of a multi-warp small eigensolver (named barriers 1
// and, between the sweeps, 2: the rest of a block may use barrier 0)
__device__ __forceinline__ void hess_bar(int nthr) { asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory"); }
__device__ __forceinline__ void sweep_bar(int nthr) { asm volatile("bar.sync 2, %0;" ::"r"(nthr) : "memory"); }

// what the leading warp of a multi-warp hess_core tells the others
constexpr int kHessWarps = 4;
struct SweepShared {
  int l[2], h[2];  // the window of each rotation list's sweep; l < 0: no more sweeps
  int ok, sym;
  double scale;
  double mx[kHessWarps];
};
// the sweeps' state: two rotation lists used in turn
template <typename Cx>
struct Sweeps {
  Cx* rot[2];
  SweepShared* ss;
  int buf;
};

// The column rotations of one sweep on NW warps: 32 rows of T per warp, then
// (the next sweep may start) 32 rows of Z per warp, the leading warp last.
template <typename Cx, int NW>
static __device__ __forceinline__ void sweep_cols(Cx* T, Cx* Z, int m, int ld, int l, int h, const Cx* rot, int warp,
                                                  int lane) {
  for (int i = 32 * warp + lane; i <= h; i += 32 * NW) cols_rows<Cx, true>(T, ld, i, l, h, rot);
  if (m > 32) sweep_bar(32 * NW);
  for (int i = 32 * (NW - 1 - warp) + lane; i < m; i += 32 * NW) cols_rows<Cx, false>(Z, ld, i, l, h, rot);
  __syncwarp();
}

template <typename Cx, int NW>
static __device__ __forceinline__ void warp_sweep(Cx* T, Cx* Z, int m, int ld, int l, int h, Cx mu, Sweeps<Cx>& sw,
                                                  int lane) {
  Cx* rot = sw.rot[sw.buf];
  // (the carries stay in registers when their count is fixed by m's range)
  if (m <= 32)
    warp_chain<Cx, 1>(T, m, ld, l, h, mu, rot, lane);
  else if (m <= 64)
    warp_chain<Cx, 2>(T, m, ld, l, h, mu, rot, lane);
  else if (m <= 128)
    warp_chain<Cx, 4>(T, m, ld, l, h, mu, rot, lane);
  else
    warp_chain<Cx, kMaxM / 32>(T, m, ld, l, h, mu, rot, lane);
  __syncwarp();
  if (lane == 0) {
    sw.ss->l[sw.buf] = l;
    sw.ss->h[sw.buf] = h;
  }
  sweep_bar(32 * NW);
  sweep_cols<Cx, NW>(T, Z, m, ld, l, h, rot, 0, lane);
  sw.buf ^= 1;
}

// the other warps' side of the leading warp's sweeps, until it ends them
template <typename Cx, int NW>
static __device__ __forceinline__ void help_sweeps(Cx* T, Cx* Z, int m, int ld, Sweeps<Cx>& sw, int warp, int lane) {
  for (;;) {
    sweep_bar(32 * NW);
    const int l = sw.ss->l[sw.buf], h = sw.ss->h[sw.buf];
    const Cx* rot = sw.rot[sw.buf];
    sw.buf ^= 1;
    if (l < 0) return;
    sweep_cols<Cx, NW>(T, Z, m, ld, l, h, rot, warp, lane);
  }
}
template <typename Cx, int NW>
static __device__ void end_sweeps(Sweeps<Cx>& sw, int lane) {
  if (lane == 0) sw.ss->l[sw.buf] = -1;
  sweep_bar(32 * NW);
  sw.buf ^= 1;
}

// Householder reduction of dense T to Hessenberg form, Z accumulating.
template <typename Cx>
static __device__ void warp_hessenberg(Cx* T, Cx* Z, Cx* v, int m, int ld, int lane) {
  using R = decltype(Cx::re);
  for (int k = 0; k + 2 < m; ++k) {
    R s = 0;
    for (int i = k + 1 + lane; i < m; i += 32) s += abs2(TT_(i, k));
    s = warp_sum_t(s);
    R a = sqrt(s);
    if (a == 0) continue;
    Cx x0 = TT_(k + 1, k);
    R ax0 = cabs_(x0);
    Cx ph = ax0 > 0 ? Cx{x0.re / ax0, x0.im / ax0} : Cx{1, 0};
    for (int i = lane; i < m; i += 32) v[i] = (i > k) ? TT_(i, k) : Cx{0, 0};
    __syncwarp();
    if (lane == 0) v[k + 1] = v[k + 1] + a * ph;
    __syncwarp();
    R vv = 0;
    for (int i = k + 1 + lane; i < m; i += 32) vv += abs2(v[i]);
    vv = warp_sum_t(vv);
    const R f = R(2) / vv;
    // T <- P T : column j (two partial sums break the dependency chain)
    for (int j = lane; j < m; j += 32) {
      Cx d0 = {0, 0}, d1 = {0, 0};
      int i = k + 1;
      for (; i + 1 < m; i += 2) {
        d0 = d0 + conj(v[i]) * TT_(i, j);
        d1 = d1 + conj(v[i + 1]) * TT_(i + 1, j);
      }
      if (i < m) d0 = d0 + conj(v[i]) * TT_(i, j);
      const Cx d = f * (d0 + d1);
      for (i = k + 1; i < m; ++i) TT_(i, j) = TT_(i, j) - d * v[i];
    }
    __syncwarp();
    // T <- T P, Z <- Z P : row i
    for (int i = lane; i < m; i += 32) {
      Cx d0 = {0, 0}, d1 = {0, 0}, e0 = {0, 0}, e1 = {0, 0};
      int j = k + 1;
      for (; j + 1 < m; j += 2) {
        d0 = d0 + TT_(i, j) * v[j];
        d1 = d1 + TT_(i, j + 1) * v[j + 1];
        e0 = e0 + ZZ_(i, j) * v[j];
        e1 = e1 + ZZ_(i, j + 1) * v[j + 1];
      }
      if (j < m) {
        d0 = d0 + TT_(i, j) * v[j];
        e0 = e0 + ZZ_(i, j) * v[j];
      }
      const Cx d = f * (d0 + d1), e = f * (e0 + e1);
      for (j = k + 1; j < m; ++j) {
        TT_(i, j) = TT_(i, j) - d * conj(v[j]);
        ZZ_(i, j) = ZZ_(i, j) - e * conj(v[j]);
      }
    }
    __syncwarp();
    for (int i = k + 2 + lane; i < m; i += 32) TT_(i, k) = Cx{0, 0};
    __syncwarp();
  }
}

// The Householder reduction on NW warps (m <= 32, all NW warps calling;
// warp 0 forms each reflector): per step, P T has one lane per column and
// the rows split over the warps (partial sums v^H T summed through shared
// memory), T P and Z P one lane per row and the columns split over the
// warps.  part: 2 NW x 32 entries of shared scratch; v: 32; fs: 1.
template <typename Cx, int NW>
static __device__ void block_hessenberg32(Cx* T, Cx* Z, Cx* v, Cx* part, decltype(Cx::re)* fs, int m, int ld,
                                          int warp, int lane) {
  using R = decltype(Cx::re);
  constexpr int nthr = NW * 32;
  const Cx zero = {0, 0};
  Cx* pa = part;            // NW x 32: P T partials, then T P partials
  Cx* pz = part + NW * 32;  // NW x 32: Z P partials
  for (int k = 0; k + 2 < m; ++k) {
    hess_bar(nthr);  // the previous step's updates are in place
    if (warp == 0) {
      const Cx xi = (lane > k && lane < m) ? TT_(lane, k) : zero;
      const R s = warp_sum_t(abs2(xi));
      const Cx x0 = shfl_c(xi, k + 1);
      R f = 0;
      Cx vi = xi;
      if (s > 0) {
        const R a = sqrt_t(s), ax0 = sqrt_t(abs2(x0));
        const Cx ph = ax0 > 0 ? Cx{x0.re / ax0, x0.im / ax0} : Cx{1, 0};
        if (lane == k + 1) vi = xi + a * ph;
        f = R(1) / (a * (a + ax0));  // 2 / |v|^2
      }
      v[lane] = vi;  // zero outside rows k + 1 .. m - 1
      if (lane == 0) *fs = f;
    }
    hess_bar(nthr);
    const R f = *fs;
    if (f == 0) continue;  // column k is reduced already (the same for every warp)
    // P T: lane j = column (j >= k), this warp's rows of k + 1 .. m - 1
    const int nr = m - k - 1, cr = (nr + NW - 1) / NW;
    const int i0 = k + 1 + warp * cr, i1 = i0 + cr < m ? i0 + cr : m;
    const bool colj = lane >= k && lane < m;
    {
      Cx w0 = zero, w1 = zero;
      if (colj) {
        int i = i0;
        for (; i + 1 < i1; i += 2) {
          w0 = cfma(conj(v[i]), TT_(i, lane), w0);
          w1 = cfma(conj(v[i + 1]), TT_(i + 1, lane), w1);
        }
        if (i < i1) w0 = cfma(conj(v[i]), TT_(i, lane), w0);
      }
      pa[warp * 32 + lane] = w0 + w1;
    }
    hess_bar(nthr);
    {
      Cx w = pa[lane];
#pragma unroll
      for (int u = 1; u < NW; ++u) w = w + pa[u * 32 + lane];
      w = f * w;
      if (colj)
        for (int i = i0; i < i1; ++i) TT_(i, lane) = (lane == k && i >= k + 2) ? zero : cfma(-v[i], w, TT_(i, lane));
    }
    hess_bar(nthr);
    // T P, Z P: lane i = row, this warp's columns of k + 1 .. m - 1
    const int j0 = k + 1 + warp * cr, j1 = j0 + cr < m ? j0 + cr : m;
    const bool rowi = lane < m;
    {
      Cx y0 = zero, y1 = zero;
      if (rowi)
        for (int j = j0; j < j1; ++j) {
          y0 = cfma(TT_(lane, j), v[j], y0);
          y1 = cfma(ZZ_(lane, j), v[j], y1);
        }
      pa[warp * 32 + lane] = y0;
      pz[warp * 32 + lane] = y1;
    }
    hess_bar(nthr);
    {
      Cx y = pa[lane], yz = pz[lane];
#pragma unroll
      for (int u = 1; u < NW; ++u) {
        y = y + pa[u * 32 + lane];
        yz = yz + pz[u * 32 + lane];
      }
      y = f * y;
      yz = f * yz;
      if (rowi)
        for (int j = j0; j < j1; ++j) {
          TT_(lane, j) = cfma(-y, conj(v[j]), TT_(lane, j));
          ZZ_(lane, j) = cfma(-yz, conj(v[j]), ZZ_(lane, j));
        }
    }
  }
  hess_bar(nthr);
}

// Complex Schur form in place; returns false when the sweep budget ran out.
template <typename Cx, int NW>
static __device__ __forceinline__ bool warp_schur(Cx* T, Cx* Z, int m, int ld, Sweeps<Cx>& sw, int lane) {
  using R = decltype(Cx::re);
  int h = m - 1, its = 0, total = 0;
  while (h > 0) {
    const int l = find_split(T, ld, h, lane);
    if (l > 0 && lane == 0) TT_(l, l - 1) = Cx{0, 0};
    __syncwarp();
    if (l == h) {
      --h;
      its = 0;
      continue;
    }
    if (++total > 30 * m) return false;
    // Wilkinson shift: the eigenvalue of the trailing 2 x 2 nearer d
    // (prescaled entries: squared moduli stay in range); every tenth sweep
    // of a window an exceptional shift d + |c|
    const Cx a = TT_(h - 1, h - 1), b = TT_(h - 1, h), c = TT_(h, h - 1), d = TT_(h, h);
    const Cx tr2 = R(0.5) * (a + d), amd = R(0.5) * (a - d);
    const Cx disc = csqrt_s(cfma(amd, amd, b * c));
    const Cx m1 = tr2 + disc, m2 = tr2 - disc;
    Cx mu = abs2(m1 - d) < abs2(m2 - d) ? m1 : m2;
    if (its > 0 && its % 10 == 0) mu = d + Cx{sqrt_t(abs2(c)), 0};
    warp_sweep<Cx, NW>(T, Z, m, ld, l, h, mu, sw, lane);
    ++its;
  }
  __syncwarp();
  return true;
}

// Hermitian tridiagonal path (the restart loop of a Hermitian operator,
// real symmetric included, whose Hessenberg matrix is Hermitian tridiagonal
// to rounding): with the diagonal unitary D of phases D_0 = 1, D_{i+1} =
// D_i e_i / |e_i| (e_i = H[i+1][i]), H = D T' D^H where T' is real
// symmetric tridiagonal with diagonal Re H[i][i] and off-diagonal |e_i|.
// d (m) and e (m - 1) of T' are real in shared memory; Z starts as D and
// accumulates the real rotations, so Z = D Q' holds the eigenvectors of H
// (and the exact shifts' Q for the restart, with T' after the shifts as the
// new H).  The implicit QR step with shift mu on the window [l, h] (Golub &
// Van Loan, Matrix Computations, Alg. 8.3.2) runs its rotation chain on
// lane 0 and records the rotations (c, s) in cs; every lane then applies
// them to one row of Z (Z <- Z G^T).  The rotation of the pair (x, y) is
// c = x / r, s = y / r (the entries are prescaled, so r^2 stays in range; a
// pair below tiny2 gives the identity).

// true when T (prescaled: largest entry in [1, 2), m x m) is Hermitian to
// rtol: the Arnoldi matrix of a Hermitian operator, whose entries beyond the
// tridiagonal band and whose departure from Hermitian symmetry come from the
// basis's loss of orthogonality (about 4e-13 of max |H| for a real n = 256
// operator with eigenvalues over three decades); they are dropped, which
// moves the Ritz values by as much, so rtol is a tenth of the residual goal
// (every result is verified against the operator)
template <typename Cx>
static __device__ bool warp_is_hermitian(const Cx* T, int m, int ld, double rtol, int lane) {
  using R = decltype(Cx::re);
  const R tol = (R)rtol;
  int bad = 0;
  for (int e = lane; e < m * m; e += 32) {
    const int r = e % m, c = e / m;
    const Cx a = TT_(r, c), b = TT_(c, r);
    if (!(abs_t(a.re - b.re) <= tol && abs_t(a.im + b.im) <= tol)) bad = 1;
  }
  return !__any_sync(0xffffffffu, bad);
}

template <typename R>
static __device__ void symtri_step(R* d, R* e, R* cs, int l, int h, R mu) {  // one lane
  R x = d[l] - mu, y = e[l];
  for (int k = l; k < h; ++k) {
    const R r2 = x * x + y * y;
    const bool ok = r2 > HessK<R>::tiny2;
    const R ir = rsqrt_t(ok ? r2 : R(1));
    const R c = ok ? x * ir : R(1), s = ok ? y * ir : R(0);
    if (k > l) e[k - 1] = ok ? r2 * ir : x;
    const R dk = d[k], dk1 = d[k + 1], ek = e[k];
    const R t1 = c * dk + s * ek, t2 = c * ek + s * dk1;
    const R t3 = c * ek - s * dk, t4 = c * dk1 - s * ek;
    d[k] = c * t1 + s * t2;
    e[k] = c * t2 - s * t1;
    d[k + 1] = c * t4 - s * t3;
    cs[2 * k] = c;
    cs[2 * k + 1] = s;
    if (k + 1 < h) {  // the bulge at (k + 2, k)
      x = e[k];
      y = s * e[k + 1];
      e[k + 1] = c * e[k + 1];
    }
  }
}

// Z <- Z G_l^T ... G_{h-1}^T, one lane per row
template <typename Cx>
static __device__ void symtri_apply_z(Cx* Z, const decltype(Cx::re)* cs, int m, int ld, int l, int h, int lane) {
  for (int i = lane; i < m; i += 32) {
    Cx zc = ZZ_(i, l);
    for (int k = l; k < h; ++k) {
      const auto c = cs[2 * k], s = cs[2 * k + 1];
      const Cx z1 = ZZ_(i, k + 1);
      ZZ_(i, k) = Cx{c * zc.re + s * z1.re, c * zc.im + s * z1.im};
      zc = Cx{c * z1.re - s * zc.re, c * z1.im - s * zc.im};
    }
    ZZ_(i, h) = zc;
  }
}

// the largest l in [1, h] with e[l-1] negligible, else 0 (all lanes)
template <typename R>
static __device__ int symtri_split(const R* d, const R* e, int h, int lane) {
  for (int base = h; base >= 1; base -= 32) {
    const int l = base - lane;
    const bool f = l >= 1 && abs_t(e[l - 1]) <= HessK<R>::eps * (abs_t(d[l - 1]) + abs_t(d[l]));
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (bal) return base - (__ffs(bal) - 1);
  }
  return 0;
}

// T (m x m, Hermitian tridiagonal) -> d, e of T'; Z (the identity on
// entry) <- D, the phases
template <typename Cx>
static __device__ void symtri_load(const Cx* T, Cx* Z, int m, int ld, decltype(Cx::re)* d, decltype(Cx::re)* e,
                                   int lane) {
  using R = decltype(Cx::re);
  for (int i = lane; i < m; i += 32) {
    d[i] = TT_(i, i).re;
    if (i + 1 < m) e[i] = sqrt_t(abs2(TT_(i + 1, i)));
  }
  __syncwarp();
  if (lane == 0) {
    Cx ph = {1, 0};
    for (int i = 0; i + 1 < m; ++i) {
      const Cx sub = TT_(i + 1, i);
      const R a = e[i];
      if (a > 0) ph = ph * Cx{sub.re / a, sub.im / a};
      ZZ_(i + 1, i + 1) = ph;
    }
  }
  __syncwarp();
}
template <typename Cx>
static __device__ void symtri_store(Cx* T, int m, int ld, const decltype(Cx::re)* d, const decltype(Cx::re)* e,
                                    int lane) {
  __syncwarp();
  for (int x = lane; x < m * m; x += 32) {
    const int r = x % m, c = x / m;
    using R = decltype(Cx::re);
    const R v = r == c ? d[r] : (r == c + 1 ? e[c] : (c == r + 1 ? e[r] : R(0)));
    TT_(r, c) = Cx{v, 0};
  }
  __syncwarp();
}

// Eigen-decomposition of the symmetric tridiagonal (d, e): d becomes the
// eigenvalues, Z accumulates the rotations; false when the sweep budget ran
// out.
template <typename Cx>
static __device__ bool warp_symtri_eig(decltype(Cx::re)* d, decltype(Cx::re)* e, decltype(Cx::re)* cs, Cx* Z, int m,
                                       int ld, int lane) {
  using R = decltype(Cx::re);
  int h = m - 1, its = 0, total = 0;
  while (h > 0) {
    const int l = symtri_split(d, e, h, lane);
    __syncwarp();
    if (l > 0 && lane == 0) e[l - 1] = 0;
    __syncwarp();
    if (l == h) {
      --h;
      its = 0;
      continue;
    }
    if (++total > 30 * m) return false;
    if (lane == 0) {
      // Wilkinson shift: the eigenvalue of the trailing 2 x 2 nearer d[h];
      // every tenth step of a window an exceptional shift d[h] + |e[h-1]|
      const R a = d[h - 1], c = d[h], b = e[h - 1];
      const R del = R(0.5) * (a - c);
      const R den = del + (del >= 0 ? R(1) : R(-1)) * sqrt_t(del * del + b * b);
      R mu = den != 0 ? c - b * b / den : c;
      if (its > 0 && its % 10 == 0) mu = c + abs_t(b);
      symtri_step(d, e, cs, l, h, mu);
    }
    __syncwarp();
    symtri_apply_z(Z, cs, m, ld, l, h, lane);
    __syncwarp();
    ++its;
  }
  return true;
}

// Eigenvectors y_q = Z u_q (q < nvec) of the upper triangular T for the
// diagonal entries ord[q]: u by back substitution, one lane per eigenvector
// (columns of U in the scratch, stride min(32, nvec)), then Y = Z U one
// lane per row.  The back substitution divides through |den|^2 (one real
// reciprocal per step; T is prescaled, so |den|^2 >= small^2 stays in
// range).  warp_backsub: one warp, the U columns of eigenvectors
// q0 .. q0 + 31.
template <typename Cx>
static __device__ void warp_backsub(const Cx* T, int m, int ld, const int* ord, int nvec, int q0, double small_d,
                                    Cx* U, int lane) {
  using R = decltype(Cx::re);
  const R small = (R)small_d, small2 = small * small;
  const Cx zero = {0, 0};
  const int W = nvec < 32 ? nvec : 32;
  const int q = q0 + lane;
  const bool act = lane < W && q < nvec;
  const int idx = act ? ord[q] : 0;
  const Cx lam = TT_(idx, idx);
  if (lane < W)
    for (int i = 0; i < m; ++i) U[i * W + lane] = (act && i == idx) ? Cx{1, 0} : zero;
  for (int i = m - 2; i >= 0; --i) {
    Cx a0 = zero, a1 = zero;
    if (lane < W) {
      int j = i + 1;
      for (; j + 1 < m; j += 2) {
        a0 = cfma(TT_(i, j), U[j * W + lane], a0);
        a1 = cfma(TT_(i, j + 1), U[(j + 1) * W + lane], a1);
      }
      if (j < m) a0 = cfma(TT_(i, j), U[j * W + lane], a0);
    }
    if (act && i < idx) {
      Cx den = TT_(i, i) - lam;
      R d2 = abs2(den);
      if (d2 < small2) {
        den = Cx{small, 0};
        d2 = small2;
      }
      const Cx ui = (-R(1) / d2) * ((a0 + a1) * conj(den));
      U[i * W + lane] = ui;
      if (cabs1(ui) > HessK<R>::big)  // rescale this column to avoid overflow
        for (int j = i; j <= idx; ++j) U[j * W + lane] = HessK<R>::unbig * U[j * W + lane];
    }
  }
}

// Y[:, q] = Z U[:, q - q0] normalised, and the estimates beta |y_q[m-1]| /
// (scale ||y_q||), for the eigenvectors q0 + c with c < nq in this warp's
// share: for m <= 32, chunks of eight columns c0 = 8 (part + nparts t), one
// lane per row, their norms summed by interleaved butterflies.  Returns the
// largest estimate over q < k of the share.
template <typename Cx>
static __device__ double warp_zu(const Cx* Z, int m, int ld, const Cx* U, int W, int q0, int nq, int k, double beta,
                                 double scale, cplx* Y, double* est, int part, int nparts, int lane) {
  using R = decltype(Cx::re);
  const Cx zero = {0, 0};
  double maxest = 0;
  if (m <= 32) {
    constexpr int CH = 8;
    const bool rin = lane < m;
    for (int c0 = CH * part; c0 < nq; c0 += CH * nparts) {
      Cx y[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) y[c] = zero;
      for (int j = 0; j < m; ++j) {
        const Cx z = rin ? ZZ_(lane, j) : zero;
#pragma unroll
        for (int c = 0; c < CH; ++c) y[c] = cfma(z, U[j * W + (c0 + c < nq ? c0 + c : c0)], y[c]);
      }
      R n2[CH];
      Cx yl[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        n2[c] = abs2(y[c]);
        yl[c] = shfl_c(y[c], m - 1);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < CH; ++c) n2[c] += __shfl_xor_sync(0xffffffffu, n2[c], o);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int qq = q0 + c0 + c;
        if (c0 + c < nq) {
          const R nrm = sqrt_t(n2[c]);
          const R inv = nrm > 0 ? R(1) / nrm : R(0);
          if (rin) Y[(long)qq * m + lane] = cx_to(inv * y[c]);
          const double e = beta * (double)sqrt_t(abs2(yl[c])) * (double)inv / scale;
          if (lane == 0) est[qq] = e;
          if (qq < k) maxest = fmax(maxest, e);
        }
      }
    }
    return maxest;
  }
  for (int c = part; c < nq; c += nparts) {
    const int qq = q0 + c;
    Cx yv[kMaxM / 32];
    R nrm = 0;
    Cx ylast = zero;
#pragma unroll
    for (int t = 0; t < kMaxM / 32; ++t) {
      const int r = lane + 32 * t;
      yv[t] = zero;
      if (r < m) {
        Cx s0 = zero, s1 = zero;
        int j = 0;
        for (; j + 1 < m; j += 2) {
          s0 = cfma(ZZ_(r, j), U[j * W + c], s0);
          s1 = cfma(ZZ_(r, j + 1), U[(j + 1) * W + c], s1);
        }
        if (j < m) s0 = cfma(ZZ_(r, j), U[j * W + c], s0);
        yv[t] = s0 + s1;
        nrm += abs2(yv[t]);
        if (r == m - 1) ylast = yv[t];
      }
    }
    nrm = sqrt(warp_sum_t(nrm));
    ylast.re = warp_sum_t(ylast.re);
    ylast.im = warp_sum_t(ylast.im);
    const R inv = nrm > 0 ? R(1) / nrm : R(0);
#pragma unroll
    for (int t = 0; t < kMaxM / 32; ++t) {
      const int r = lane + 32 * t;
      if (r < m) Y[(long)qq * m + r] = cx_to(inv * yv[t]);
    }
    const double e = beta * (double)cabs_(ylast) * (double)inv / scale;
    if (lane == 0) est[qq] = e;
    if (qq < k) maxest = fmax(maxest, e);
  }
  return maxest;
}

// Shared scratch of block_hessenberg32.
template <typename Cx, int NW>
struct HouseShared {
  Cx v[32];
  Cx part[2 * NW * 32];
  decltype(Cx::re) f;
};

// The body of k_hess on NW >= 2 warps (tid = 0 .. 32 NW - 1 of the calling
// threads), with its workspaces passed in: T, Z (leading dimension
// hess_ld(m), m columns each), u (m), key (m), ord (m), scratch
// (hess_scratch_cplx(m); 2 m + 2 + m max(2, min(nvec, 32)) of it are used).
// SH: T, Z and the scratch lie in shared memory.
// Callable from any kernel by NW full warps, with shared scratch ss and, for
// a dense input of m <= 32, hs; the outputs in `a` may point to shared or
// global memory.  The sweeps' column rotations and, for m <= 32, the
// Householder reduction and the product Y = Z U run on all warps; the rotation
// chains, the sort and the back substitutions on warp 0.
template <typename Cx, int NW, bool SH = true>
static __device__ void hess_core(const HessArgs& a, Cx* T, Cx* Z, Cx* u, double* key, int* ord, Cx* scratch,
                                 int tid, SweepShared* ss, HouseShared<Cx, NW>* hs = nullptr) {
  if constexpr (SH) {
    T = as_shared(T);
    Z = as_shared(Z);
    scratch = as_shared(scratch);
  }
  using R = decltype(Cx::re);
  constexpr int nthr = NW * 32;
  const int lane = tid & 31, warp = tid >> 5;
  const int m = a.m, k = a.k, ld = hess_ld(m);
  const long mm = (long)m * m;
  DevState* st = a.st;
  Cx* rot = scratch;           // 2 m
  Cx* U = scratch + 2 * m + 2; // m x 32; the second rotation list during the sweeps
  Sweeps<Cx> sw{{rot, U}, ss, 0};

  // T = sig H with sig a power of two that puts the largest |re| or |im| of
  // H in [1, 2): exact, and the Schur sweeps' rotations and shifts then need
  // no overflow / underflow branches (givens_s, csqrt_s).  Values leave
  // hess_core unscaled (times isig).  (Every warp finds the same maximum.)
  double mx = 0;
  for (long i = lane; i < mm; i += 32) mx = fmax(mx, fmax(fabs(a.Hin[i].re), fabs(a.Hin[i].im)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  int ex = 0;
  if (mx > 0 && mx <= 1.7e308) frexp(mx, &ex);  // mx = f 2^ex, f in [0.5, 1)
  ex = ex > 1000 ? 1000 : (ex < -1000 ? -1000 : ex);
  const double sig = ldexp(1.0, 1 - ex), isig = ldexp(1.0, ex - 1);
  for (long i = tid; i < mm; i += nthr) {
    const int r = (int)(i % m), c = (int)(i / m);
    TT_(r, c) = cx_from<Cx>(sig * a.Hin[i]);
    ZZ_(r, c) = (r == c) ? Cx{1, 0} : Cx{0, 0};
  }
  hess_bar(nthr);
  if (a.dense && m <= 32 && hs) {
    block_hessenberg32<Cx, NW>(T, Z, hs->v, hs->part, &hs->f, m, ld, warp, lane);
  } else if (a.dense) {
    if (warp == 0) warp_hessenberg(T, Z, u, m, ld, lane);
    hess_bar(nthr);
  }
  const int nvec = a.nvec > k ? (a.nvec < m ? a.nvec : m) : k;
  const int W = nvec < 32 ? nvec : 32;
  double scale = 0, small = 0;
  const double beta = a.use_beta ? sqrt(st->fnorm2) : a.beta;
  // Hermitian Hessenberg input: the tridiagonal path (d, e in the
  // eigenvector scratch, the rotations in rot)
  R* sd = reinterpret_cast<R*>(U);
  R* se = sd + m;
  R* scs = reinterpret_cast<R*>(rot);
  bool sym = false;
  if (warp == 0) {
    sym = !a.dense && a.tol > 0 && warp_is_hermitian(T, m, ld, 0.1 * a.tol, lane);
    if (sym && lane == 0) st->symtri += 1;
    if (lane == 0) ss->sym = sym;
    sweep_bar(nthr);
    bool ok;
    if (sym) {
      symtri_load(T, Z, m, ld, sd, se, lane);
      ok = warp_symtri_eig(sd, se, scs, Z, m, ld, lane);
      if (ok) {
        for (int i = lane; i + 1 < m; i += 32) se[i] = 0;
        symtri_store(T, m, ld, sd, se, lane);
      }
    } else {
      ok = warp_schur<Cx, NW>(T, Z, m, ld, sw, lane);
      end_sweeps<Cx, NW>(sw, lane);
    }
    if (!ok && lane == 0) {
      st->status |= 2;
      st->converged = 0;
    }
    if (lane == 0) ss->ok = ok;
    if (ok) {
      // sort order of diag(T)
      for (int i = lane; i < m; i += 32) {
        double kv = sort_key(cx_to(TT_(i, i)), a.which);
        key[i] = (kv != kv) ? INFINITY : kv;  // NaN sorts last; ranks stay a permutation
      }
      __syncwarp();
      for (int i = lane; i < m; i += 32) {
        int r = 0;
        for (int j = 0; j < m; ++j) r += (key[j] < key[i]) || (key[j] == key[i] && j < i);
        ord[r] = i;
      }
      __syncwarp();
      for (int q = lane; q < m; q += 32) {
        a.order[q] = ord[q];
        a.ritz[q] = isig * cx_to(TT_(ord[q], ord[q]));
      }
      // max |theta| over the wanted set, unscaled
      for (int q = 0; q < k; ++q) scale = fmax(scale, (double)cabs_(TT_(ord[q], ord[q])));
      scale *= isig;
      if (scale == 0) scale = 1;
      double tnorm = 0;
      for (int i = lane; i < m; i += 32) tnorm = fmax(tnorm, (double)cabs_(TT_(i, i)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
      small = (double)HessK<R>::eps * (tnorm > 0 ? tnorm : 1.0);
      warp_backsub(T, m, ld, ord, nvec, 0, small, U, lane);
      if (lane == 0) ss->scale = scale;
    }
    __syncwarp();
  } else {
    sweep_bar(nthr);
    sym = ss->sym;
    if (!sym) help_sweeps<Cx, NW>(T, Z, m, ld, sw, warp, lane);
  }
  double maxest = 0;
  hess_bar(nthr);
  if (!ss->ok) return;  // the Schur sweeps ran out (status set)
  scale = ss->scale;
  // eigenvectors of the first nvec Ritz values (the wanted k and optional
  // guard vectors), for m <= 32 on all warps
  if (m <= 32) {
    maxest = warp_zu(Z, m, ld, U, W, 0, nvec, k, beta, scale, a.Y, a.est, warp, NW, lane);
  } else if (warp == 0) {
    for (int q0 = 0; q0 < nvec; q0 += 32) {
      if (q0 > 0) {
        warp_backsub(T, m, ld, ord, nvec, q0, small, U, lane);
        __syncwarp();
      }
      const int nq = (nvec - q0) < W ? (nvec - q0) : W;
      maxest = fmax(maxest, warp_zu(Z, m, ld, U, W, q0, nq, k, beta, scale, a.Y, a.est, 0, 1, lane));
      __syncwarp();
    }
  }
  if (lane == 0) ss->mx[warp] = maxest;
  hess_bar(nthr);
  for (int w = 0; w < NW; ++w) maxest = fmax(maxest, ss->mx[w]);
  const int conv = maxest <= a.tol;
  if (tid == 0) {
    st->converged = conv;
    st->scale = scale;
    st->maxest = maxest;
  }
  if (conv || !a.do_shift) return;

  // exact shifts on H with the unwanted Ritz values (kept in u[] before T
  // is reloaded with H)
  if (warp == 0) {
    __syncwarp();
    for (int q = lane; q < m; q += 32) u[q] = TT_(ord[q], ord[q]);
    __syncwarp();
  }
  hess_bar(nthr);
  for (long i = tid; i < mm; i += nthr) {
    const int r = (int)(i % m), c = (int)(i / m);
    TT_(r, c) = cx_from<Cx>(sig * a.Hin[i]);
    ZZ_(r, c) = (r == c) ? Cx{1, 0} : Cx{0, 0};
  }
  hess_bar(nthr);
  if (warp != 0) {
    if (!sym) help_sweeps<Cx, NW>(T, Z, m, ld, sw, warp, lane);
    hess_bar(nthr);
    return;
  }
  if (sym) {  // the same exact shifts as implicit symmetric tridiagonal steps
    symtri_load(T, Z, m, ld, sd, se, lane);
    for (int q = a.keep; q < m; ++q) {
      const R mu = u[q].re;
      int hb = m - 1;
      while (hb > 0) {
        const int l = symtri_split(sd, se, hb, lane);
        __syncwarp();
        if (l > 0 && lane == 0) se[l - 1] = 0;
        __syncwarp();
        if (l < hb) {
          if (lane == 0) symtri_step(sd, se, scs, l, hb, mu);
          __syncwarp();
          symtri_apply_z(Z, scs, m, ld, l, hb, lane);
          __syncwarp();
        }
        hb = l - 1;
      }
    }
    symtri_store(T, m, ld, sd, se, lane);
  } else {
    for (int q = a.keep; q < m; ++q) {
      Cx mu = u[q];
      if (a.real_shifts) mu.im = 0;
      int hb = m - 1;
      while (hb > 0) {
        const int l = find_split(T, ld, hb, lane);
        if (l > 0 && lane == 0) TT_(l, l - 1) = Cx{0, 0};
        __syncwarp();
        if (l < hb) warp_sweep<Cx, NW>(T, Z, m, ld, l, hb, mu, sw, lane);
        hb = l - 1;
      }
    }
    end_sweeps<Cx, NW>(sw, lane);
  }
  hess_bar(nthr);  // the other warps' rows of Z are in place
  if (lane == 0) {
    st->beta_hat = isig * cx_to(TT_(a.keep, a.keep - 1));
    st->sigma = cx_to(ZZ_(m - 1, a.keep - 1));
    st->keep = a.keep;
    st->spike = 0;
  }
  for (long i = lane; i < mm; i += 32) {
    const int r = (int)(i % m), c = (int)(i / m);
    a.Hout[i] = (r < a.keep && c < a.keep) ? isig * cx_to(TT_(r, c)) : cplx{0, 0};
    a.Qout[i] = cx_to(ZZ_(r, c));
  }
}

// threads of k_hess / k_hess_f32
__host__ __device__ inline int hess_threads(int) { return 32 * kHessWarps; }

// dynamic shared memory (or a.gws): T, Z, scratch of the working type Cx;
// launched with hess_threads(m) threads
template <typename Cx>
static __device__ void hess_kernel_body(const HessArgs& a, unsigned char* dyn) {
  __shared__ Cx u[kMaxM];
  __shared__ double key[kMaxM];
  __shared__ int ord[kMaxM];
  __shared__ SweepShared ss;
  __shared__ HouseShared<Cx, kHessWarps> hs;
  const size_t tz = (size_t)hess_ld(a.m) * a.m;
  if (Cx* T = reinterpret_cast<Cx*>(a.gws))
    hess_core<Cx, kHessWarps, false>(a, T, T + tz, u, key, ord, T + 2 * tz, threadIdx.x, &ss, &hs);
  else if (Cx* S = reinterpret_cast<Cx*>(dyn))
    hess_core<Cx, kHessWarps>(a, S, S + tz, u, key, ord, S + 2 * tz, threadIdx.x, &ss, &hs);
}

// FP64 working arithmetic (the restart loop and the refinement)
static __global__ void __launch_bounds__(32 * kHessWarps) k_hess(HessArgs a) {
  extern __shared__ __align__(16) unsigned char hess_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  if (a.skip && *(volatile const int*)a.skip) return;
  hess_kernel_body<cplx>(a, hess_dyn);
}

// FP32 working arithmetic, FP64 inputs and outputs: the Rayleigh-Ritz checks
// of the FP32-class phase (whose Ritz vectors are FP32-accurate at best);
// dynamic shared memory hess_ws_cplx(m) * sizeof(cplxf)
static __global__ void __launch_bounds__(32 * kHessWarps) k_hess_f32(HessArgs a) {
  extern __shared__ __align__(16) unsigned char hess_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  hess_kernel_body<cplxf>(a, hess_dyn);
}

#undef TT_
#undef ZZ_

// Eigenpairs of a nearly upper-triangular T (m x m complex, column-major,
// m <= 32): the Rayleigh quotient of an orthonormalised basis of Ritz vectors
// ordered like their values, whose strictly lower part is of the size of the
// Ritz vectors' errors.  k_eig_near_tri: one CTA of one warp per pair q
// (grid m, each pair on its own SM): Rayleigh quotient iteration from v =
// e_q, sigma = T(q,q) (LU with partial pivoting of T - sigma I, a zero pivot
// replaced by eps ||T||_F; v <- (T - sigma I)^-1 v normalised; sigma <- v^H
// T v), at most kNtIters steps, until ||T v - sigma v|| <= 16 eps ||T||_F;
// the pair goes to the scratch (V column q at V + q m, th[q]) and ok[0] is
// cleared when its residual is above 64 eps ||T||_F.  k_eig_near_tri_finish
// (one warp, after it): accepted when ok[0] is set and the values are
// pairwise apart by more than 1e-9 max |theta|; then ritz / Y / order are
// written in the ArnUtils order of `which` (as k_hess writes them, Y column
// q at Y + q m, unit 2-norm) and *delivered = 1; otherwise *delivered = 0
// and nothing else is written (k_hess follows with skip = delivered).
// ok[0] is set again for the next call (it must hold 1 before the first).
constexpr int kNtIters = 4;
__host__ __device__ inline int nt_ld(int m) { return m + 1; }
// dynamic shared memory of k_eig_near_tri: T, M (m x LD), x, t, the pivots'
// reciprocals (m each), pivot rows
__host__ __device__ inline size_t nt_smem_bytes(int m) {
  return sizeof(cplx) * (2 * (size_t)m * nt_ld(m) + 3 * (size_t)m) + sizeof(int) * (size_t)m;
}

static __global__ void __launch_bounds__(32) k_eig_near_tri(const cplx* __restrict__ Tin, int m, cplx* V, cplx* th,
                                                            int* ok) {
  extern __shared__ __align__(16) unsigned char nt_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  const int LD = nt_ld(m);
  cplx* T = reinterpret_cast<cplx*>(nt_dyn);  // m x LD
  cplx* M = T + (size_t)m * LD;               // m x LD
  cplx* x = M + (size_t)m * LD;               // m
  cplx* t = x + m;                            // m
  cplx* dinv = t + m;                         // m: reciprocals of U's diagonal
  int* pv = reinterpret_cast<int*>(dinv + m); // m
  const int lane = threadIdx.x, q = blockIdx.x;
  if (m < 1 || m > 32 || q >= m) return;
  // T scaled by the power of two that puts its largest |re| or |im| in
  // [1, 2) (exact): the pivots' squared moduli below stay in range; the
  // value is unscaled on output
  double mx = 0;
  for (int e = lane; e < m * m; e += 32) mx = fmax(mx, fmax(fabs(Tin[e].re), fabs(Tin[e].im)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  int ex = 0;
  if (mx > 0 && mx <= 1.7e308) frexp(mx, &ex);
  ex = ex > 1000 ? 1000 : (ex < -1000 ? -1000 : ex);
  const double sig = ldexp(1.0, 1 - ex), isig = ldexp(1.0, ex - 1);
  for (int e = lane; e < m * m; e += 32) T[(e % m) + (e / m) * LD] = sig * Tin[e];
  __syncwarp();
  double fro = 0;
  for (int e = lane; e < m * m; e += 32) fro += abs2(T[(e % m) + (e / m) * LD]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
  fro = sqrt(fro);
  const double eps = 2.220446049250313e-16;
  const double tiny = eps * (fro > 0 ? fro : 1.0);
  {
    cplx sigma = T[q + q * LD], thq = {0, 0};
    double rq = 1e300;
    for (int i = lane; i < m; i += 32) x[i] = cplx{i == q ? 1.0 : 0.0, 0.0};
    __syncwarp();
    for (int itr = 0; itr < kNtIters && !(rq <= 16 * eps * fro); ++itr) {
      for (int e = lane; e < m * m; e += 32) {
        const int r = e % m, c = e / m;
        M[r + c * LD] = T[r + c * LD] - (r == c ? sigma : cplx{0, 0});
      }
      __syncwarp();
      // LU with partial pivoting, lane = column
      for (int k = 0; k < m; ++k) {
        double best = -1;
        int bi = k;
        for (int i = k + lane; i < m; i += 32) {
          const double v = abs2(M[i + k * LD]);
          if (v > best) {
            best = v;
            bi = i;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
          }
        }
        if (lane == 0) pv[k] = bi;
        for (int c = lane; c < m; c += 32) {  // swap rows k and bi
          const cplx tmp = M[k + c * LD];
          M[k + c * LD] = M[bi + c * LD];
          M[bi + c * LD] = tmp;
        }
        __syncwarp();
        // the pivot (a zero one replaced by tiny) and its reciprocal
        // conj(p) / |p|^2, kept for the back substitution
        cplx pk = M[k + k * LD];
        double p2 = abs2(pk);
        if (!(p2 >= tiny * tiny)) {
          pk = cplx{tiny, 0};
          p2 = tiny * tiny;
        }
        const cplx inv = (1.0 / p2) * conj(pk);
        __syncwarp();
        if (lane == 0) {
          M[k + k * LD] = pk;
          dinv[k] = inv;
        }
        for (int i = k + 1 + lane; i < m; i += 32) M[i + k * LD] = M[i + k * LD] * inv;  // multipliers
        __syncwarp();
        for (int c = k + 1 + lane; c < m; c += 32) {
          const cplx ukc = M[k + c * LD];
          for (int i = k + 1; i < m; ++i) M[i + c * LD] = M[i + c * LD] - M[i + k * LD] * ukc;
        }
        __syncwarp();
      }
      // x <- (T - sigma I)^-1 x, normalised: lane i holds x_i; the row
      // swaps, then L y = P b and U x = y column by column (one shuffle of
      // the finished entry per column)
      cplx xv = lane < m ? x[lane] : cplx{0, 0};
      for (int k = 0; k < m; ++k) {
        const int r = pv[k];
        const cplx xk = shfl_c(xv, k), xr = shfl_c(xv, r);
        if (lane == k) xv = xr;
        else if (lane == r) xv = xk;
      }
      for (int j = 0; j + 1 < m; ++j) {
        const cplx xj = shfl_c(xv, j);
        if (lane > j && lane < m) xv = xv - M[lane + j * LD] * xj;
      }
      for (int i = m - 1; i >= 0; --i) {
        if (lane == i) xv = xv * dinv[i];
        const cplx xi = shfl_c(xv, i);
        if (lane < i) xv = xv - M[lane + i * LD] * xi;
      }
      double nrm = abs2(xv);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
      nrm = sqrt(nrm);
      const double sc = nrm > 0 ? 1.0 / nrm : 0.0;
      if (lane < m) x[lane] = sc * xv;
      __syncwarp();
      // Rayleigh quotient (the next shift) and residual ||T x - theta x||
      for (int i = lane; i < m; i += 32) {
        cplx acc = {0, 0};
        for (int j = 0; j < m; ++j) acc = acc + T[i + j * LD] * x[j];
        t[i] = acc;
      }
      __syncwarp();
      thq = cplx{0, 0};
      for (int i = lane; i < m; i += 32) thq = thq + conj(x[i]) * t[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        thq.re += __shfl_xor_sync(0xffffffffu, thq.re, o);
        thq.im += __shfl_xor_sync(0xffffffffu, thq.im, o);
      }
      double r2 = 0;
      for (int i = lane; i < m; i += 32) r2 += abs2(t[i] - thq * x[i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
      rq = sqrt(r2);
      sigma = thq;
    }
    for (int i = lane; i < m; i += 32) V[i + (size_t)q * m] = x[i];
    if (lane == 0) {
      th[q] = isig * thq;
      if (!(rq <= 64 * eps * fro)) ok[0] = 0;
    }
  }
}

static __global__ void __launch_bounds__(32) k_eig_near_tri_finish(int m, int which, const cplx* __restrict__ V,
                                                                   const cplx* __restrict__ th, int* ok, cplx* ritz,
                                                                   cplx* Y, int* order, int* delivered) {
  __shared__ double key[32];
  __shared__ int ord[32];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  const int lane = threadIdx.x;
  if (m < 1 || m > 32) return;
  // distinct values, then the ArnUtils order
  double tmax = 0;
  for (int q = lane; q < m; q += 32) tmax = fmax(tmax, cabs_(th[q]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
  int bad = 0;
  for (int e = lane; e < m * m; e += 32) {
    const int q = e % m, r = e / m;
    if (q < r && !(cabs_(th[q] - th[r]) > 1e-9 * tmax)) bad = 1;
  }
  bad = __any_sync(0xffffffffu, bad);
  for (int i = lane; i < m; i += 32) {
    const double kv = sort_key(th[i], which);
    key[i] = (kv != kv) ? INFINITY : kv;
  }
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    int r = 0;
    for (int j = 0; j < m; ++j) r += (key[j] < key[i]) || (key[j] == key[i] && j < i);
    ord[r] = i;
  }
  __syncwarp();
  const int good = ok[0] && !bad;
  __syncwarp();
  if (lane == 0) {
    *delivered = good;
    ok[0] = 1;
  }
  if (!good) return;
  for (int q = lane; q < m; q += 32) {
    ritz[q] = th[ord[q]];
    order[q] = ord[q];
  }
  for (int e = lane; e < m * m; e += 32) {
    const int i = e % m, q = e / m;
    Y[i + (size_t)q * m] = V[i + (size_t)ord[q] * m];
  }
}

}  // namespace oapb
