// Arnoldi steps j0 .. m - 1 of the plain FP64 restart loop on a dense
// operator, one cooperative launch per restart cycle
// (executeArnoldiFactorization, ArnoldiProcedures.cpp:407-461).
//
// What bounds a step on an operator of a few thousand rows is not the
// operator's bytes but the chain of dependent kernels: the per-step path
// launches eleven (breakdown, normalise, matvec, twice project / reduce /
// update / finalise) that take 2 - 6 us each and wait for one another.  Here
// every CTA owns a block of rows of the operator and of the basis for the
// whole cycle: its basis rows stay in shared memory, the projections and the
// update are local to the rows, and a step needs two grid barriers, one for
// the projections' sum (every CTA adds the CTAs' partials itself, in CTA
// order, so the result is deterministic and the same everywhere) and one for
// the new residual vector and its norm.  The reorthogonalisation pass costs
// two more, only when the DGKS test asks for it.  The restart's V <- V Q and
// f <- v beta_hat + f sigma are local to the rows too and open the cycle.
//
// The rows of the operator come from shared memory when they fit beside the
// rest (n up to about 1700 real, 1200 complex on 148 CTAs), loaded once per
// cycle, else from L2 / HBM with 16-byte loads (8-byte for odd n, whose rows
// are not 16-byte aligned).  A warp takes a pair of rows times a column
// segment; the segment count evens the pairs out over the 16 warps.
//
// Measured (B200, whole step): real n = 2048, m = 24: 35 us on the per-step
// kernels, 13.4 us here; complex n = 3001, m = 32: 93 us, 37 us; complex
// n = 6000, m = 48 (576 MB per pass, HBM-bound): 169 us, 101 us.
//
// Every wait is bounded (2 s): a barrier that runs out sets bit 1 of
// DevState::status and the CTA returns.
#include "cycle.cuh"

#include <algorithm>

namespace oapb {
namespace {

constexpr int kCyThreads = 512;
constexpr int kCyWarps = kCyThreads / 32;
constexpr int kCyMaxM = 128;
constexpr int kCyGroups = 8;  // row groups of the projections
constexpr int kCyMaxSegs = 8;
constexpr int kCyPre = 4;  // values of f per thread loaded with the norm's partials
constexpr uint64_t kCyLimitNs = 2000000000ull;

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// operator loads: read once per step, not kept in L1
__device__ __forceinline__ double2 ld_op2(const double* p) {
  double2 v;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_op1(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// Grid barrier on a counter that only grows during the launch: the k-th
// barrier waits for k gridDim.x arrivals.  One thread arrives (release, which
// with the CTA barrier before it covers the other threads' writes) and polls
// (acquire); returns false when the wait ran out.
__device__ bool grid_bar(unsigned* bar, unsigned& target, int* flag) {
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    unsigned v;
    int ok = 1;
    uint64_t t0 = 0;
    for (unsigned it = 0;; ++it) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) break;
      if ((it & 255u) == 255u) {
        const uint64_t t = now_ns();
        if (!t0) t0 = t;
        if (t - t0 > kCyLimitNs) {
          ok = 0;
          break;
        }
      }
    }
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

// shared memory of one CTA
template <bool C>
struct CySmem {
  double *xr, *xi;        // n (or rows x (m + 1)): the current basis vector / restart scratch
  double *vr, *vi;        // rows x ld basis rows
  double *wr, *wi, *fr, *fi;  // rows
  cplx *h, *s, *red;      // m + 1, m + 1, groups x (m + 1)
  double* seg;            // rows x segs x 2 matvec partials
  double* wsum;           // warps
  double* ar;             // rows x n operator rows (resident), planes one after the other
  int* flag;
};

__host__ __device__ inline int cy_ld(int m) { return (m + 1) | 1; }
__host__ __device__ inline long cy_xlen(int n, int rows, int m) {
  const long a = n, b = (long)rows * (m + 1);
  return ((a > b ? a : b) + 1) & ~1L;
}

template <bool C>
__host__ __device__ inline size_t cy_carve(char* base, int n, int m, int rows, int segs, bool res, CySmem<C>* S) {
  size_t o = 0;
  const int P = C ? 2 : 1;
  auto take = [&](size_t b) {
    char* p = base + o;
    o += (b + 15) & ~(size_t)15;
    return p;
  };
  const size_t xl = sizeof(double) * (size_t)cy_xlen(n, rows, m), vl = sizeof(double) * (size_t)rows * cy_ld(m),
               rl = sizeof(double) * (size_t)rows;
  CySmem<C> T;
  T.xr = (double*)take(xl);
  T.xi = C ? (double*)take(xl) : nullptr;
  T.vr = (double*)take(vl);
  T.vi = C ? (double*)take(vl) : nullptr;
  T.wr = (double*)take(rl);
  T.wi = C ? (double*)take(rl) : nullptr;
  T.fr = (double*)take(rl);
  T.fi = C ? (double*)take(rl) : nullptr;
  T.h = (cplx*)take(sizeof(cplx) * (m + 1));
  T.s = (cplx*)take(sizeof(cplx) * (m + 1));
  T.red = (cplx*)take(sizeof(cplx) * kCyGroups * (m + 1));
  T.seg = (double*)take(sizeof(double) * 2 * (size_t)rows * segs);
  T.wsum = (double*)take(sizeof(double) * kCyWarps);
  T.flag = (int*)take(sizeof(int));
  T.ar = (double*)take(res ? sizeof(double) * P * (size_t)rows * n : 0);
  if (S) *S = T;
  return o;
}

template <bool C, bool RES, bool VEC>
struct Cycle {
  const CycleArgs& a;
  CySmem<C> S;
  int n, m, ld, nr, segs;
  long r0;
  unsigned target = 0;
  int tid, warp, lane;
  double pr[kCyPre];

  // w = A x on the CTA's rows (x in shared memory)
  __device__ void matvec() {
    const int pairs = (nr + 1) >> 1, items = pairs * segs;
    const int sw = ((n + segs - 1) / segs + 63) & ~63;  // columns of a segment
    for (int it = warp; it < items; it += kCyWarps) {
      const int p = it / segs, sg = it - p * segs;
      const int ra = 2 * p, rb = ra + 1 < nr ? ra + 1 : ra;
      const int c0 = sg * sw, c1 = c0 + sw < n ? c0 + sw : n;
      const double* A0 = RES ? S.ar + (long)ra * n : a.are + (r0 + ra) * n;
      const double* A1 = RES ? S.ar + (long)rb * n : a.are + (r0 + rb) * n;
      const double* B0 = !C ? nullptr : RES ? S.ar + (long)(nr + ra) * n : a.aim + (r0 + ra) * n;
      const double* B1 = !C ? nullptr : RES ? S.ar + (long)(nr + rb) * n : a.aim + (r0 + rb) * n;
      double s0 = 0, s1 = 0, t0 = 0, t1 = 0;
      if (VEC) {
#pragma unroll 4
        for (int c = c0 + 2 * lane; c < c1; c += 64) {
          const double2 x = *(const double2*)(S.xr + c);
          const double2 p0 = RES ? *(const double2*)(A0 + c) : ld_op2(A0 + c);
          const double2 p1 = RES ? *(const double2*)(A1 + c) : ld_op2(A1 + c);
          s0 = fma(p0.x, x.x, s0);
          s1 = fma(p1.x, x.x, s1);
          s0 = fma(p0.y, x.y, s0);
          s1 = fma(p1.y, x.y, s1);
          if (C) {
            const double2 y = *(const double2*)(S.xi + c);
            const double2 q0 = RES ? *(const double2*)(B0 + c) : ld_op2(B0 + c);
            const double2 q1 = RES ? *(const double2*)(B1 + c) : ld_op2(B1 + c);
            s0 = fma(-q0.x, y.x, s0);
            s1 = fma(-q1.x, y.x, s1);
            s0 = fma(-q0.y, y.y, s0);
            s1 = fma(-q1.y, y.y, s1);
            t0 = fma(p0.x, y.x, fma(q0.x, x.x, t0));
            t1 = fma(p1.x, y.x, fma(q1.x, x.x, t1));
            t0 = fma(p0.y, y.y, fma(q0.y, x.y, t0));
            t1 = fma(p1.y, y.y, fma(q1.y, x.y, t1));
          }
        }
      } else {
#pragma unroll 4
        for (int c = c0 + lane; c < c1; c += 32) {
          const double x = S.xr[c];
          const double p0 = RES ? A0[c] : ld_op1(A0 + c), p1 = RES ? A1[c] : ld_op1(A1 + c);
          s0 = fma(p0, x, s0);
          s1 = fma(p1, x, s1);
          if (C) {
            const double y = S.xi[c];
            const double q0 = RES ? B0[c] : ld_op1(B0 + c), q1 = RES ? B1[c] : ld_op1(B1 + c);
            s0 = fma(-q0, y, s0);
            s1 = fma(-q1, y, s1);
            t0 = fma(p0, y, fma(q0, x, t0));
            t1 = fma(p1, y, fma(q1, x, t1));
          }
        }
      }
      s0 = warp_sum(s0);
      s1 = warp_sum(s1);
      if (C) {
        t0 = warp_sum(t0);
        t1 = warp_sum(t1);
      }
      if (lane == 0) {
        S.seg[2 * (ra * segs + sg)] = s0;
        if (C) S.seg[2 * (ra * segs + sg) + 1] = t0;
        if (rb != ra) {
          S.seg[2 * (rb * segs + sg)] = s1;
          if (C) S.seg[2 * (rb * segs + sg) + 1] = t1;
        }
      }
    }
    __syncthreads();
    for (int r = tid; r < nr; r += kCyThreads) {
      double s = 0, t = 0;
      for (int g = 0; g < segs; ++g) {
        s += S.seg[2 * (r * segs + g)];
        if (C) t += S.seg[2 * (r * segs + g) + 1];
      }
      S.wr[r] = s;
      if (C) S.wi[r] = t;
    }
    __syncthreads();
  }

  // dst[i] = sum over all rows of conj(V_i) x, i < nvec (x: the CTA's rows);
  // one grid barrier
  __device__ bool project(const double* xr, const double* xi, int nvec, cplx* dst) {
    const int g = tid / (kCyThreads / kCyGroups), i0 = tid % (kCyThreads / kCyGroups);
    for (int i = i0; i < nvec; i += kCyThreads / kCyGroups) {
      double p = 0, q = 0;
      for (int r = g; r < nr; r += kCyGroups) {
        const double v = S.vr[r * ld + i], x = xr[r];
        p = fma(v, x, p);
        if (C) {
          const double u = S.vi[r * ld + i], y = xi[r];
          p = fma(u, y, p);
          q = fma(v, y, fma(-u, x, q));
        }
      }
      S.red[g * (m + 1) + i] = cplx{p, q};
    }
    __syncthreads();
    const int G = gridDim.x;
    for (int i = tid; i < nvec; i += kCyThreads) {
      cplx t = S.red[i];
#pragma unroll
      for (int u = 1; u < kCyGroups; ++u) t = t + S.red[u * (m + 1) + i];
      if (C)
        __stcg((double2*)a.part + (long)i * G + blockIdx.x, make_double2(t.re, t.im));
      else
        __stcg((double*)a.part + (long)i * G + blockIdx.x, t.re);
    }
    if (!grid_bar(a.bar, target, S.flag)) return false;
    // warp w adds the CTAs' partials of vectors w, w + 16, ...: four vectors'
    // loads in flight together
    for (int b = warp; b < nvec; b += 4 * kCyWarps) {
      double p[4] = {0, 0, 0, 0}, q[4] = {0, 0, 0, 0};
      for (int c = lane; c < G; c += 32) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = b + u * kCyWarps;
          if (i < nvec) {
            if (C) {
              const double2 t = __ldcg((const double2*)a.part + (long)i * G + c);
              p[u] += t.x;
              q[u] += t.y;
            } else {
              p[u] += __ldcg((const double*)a.part + (long)i * G + c);
            }
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          p[u] += __shfl_xor_sync(0xffffffffu, p[u], o);
          if (C) q[u] += __shfl_xor_sync(0xffffffffu, q[u], o);
        }
      if (lane == 0)
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (b + u * kCyWarps < nvec) dst[b + u * kCyWarps] = cplx{p[u], q[u]};
    }
    __syncthreads();
    return true;
  }

  // the CTA's share of ||f||^2 (one value per thread) -> fpart
  __device__ void norm_partial(double s) {
    s = warp_sum(s);
    if (lane == 0) S.wsum[warp] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0;
#pragma unroll
      for (int w = 0; w < kCyWarps; ++w) t += S.wsum[w];
      __stcg(a.fpart + blockIdx.x, t);
    }
  }
  // ||f||^2 from every CTA's share (after a grid barrier; every warp adds
  // them in the same order).  The first values of f this thread will scale
  // into x are loaded beside them, so one trip to L2 covers both (real
  // operators: the complex ones have no registers to spare).
  __device__ double norm2() {
#pragma unroll
    for (int u = 0; u < (C ? 0 : kCyPre); ++u) {
      const int i = tid + u * kCyThreads;
      if (i < n) {
        pr[u] = __ldcg(a.fre + i);
      }
    }
    double t = 0;
    for (int c = lane; c < (int)gridDim.x; c += 32) t += __ldcg(a.fpart + c);
    return warp_sum(t);
  }

  // f = src - V coef on the CTA's rows, to shared and global memory, and its
  // norm; one grid barrier.  Eight lanes per row.
  __device__ bool update(const double* sr, const double* si, int nvec, const cplx* coef, double& f2) {
    double s2 = 0;
    const int sub = tid & 7;
    for (int rb = 0; rb < nr; rb += kCyThreads / 8) {
      const int r = rb + (tid >> 3);
      double p = 0, q = 0;
      if (r < nr)
        for (int i = sub; i < nvec; i += 8) {
          const double v = S.vr[r * ld + i];
          const cplx c = coef[i];
          p = fma(v, c.re, p);
          if (C) {
            const double u = S.vi[r * ld + i];
            p = fma(-u, c.im, p);
            q = fma(v, c.im, fma(u, c.re, q));
          }
        }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        p += __shfl_xor_sync(0xffffffffu, p, o);
        if (C) q += __shfl_xor_sync(0xffffffffu, q, o);
      }
      if (sub == 0 && r < nr) {
        const double x = sr[r] - p;
        S.fr[r] = x;
        __stcg(a.fre + r0 + r, x);
        s2 = fma(x, x, s2);
        if (C) {
          const double y = si[r] - q;
          S.fi[r] = y;
          __stcg(a.fim + r0 + r, y);
          s2 = fma(y, y, s2);
        }
      }
    }
    norm_partial(s2);
    if (!grid_bar(a.bar, target, S.flag)) return false;
    f2 = norm2();
    return true;
  }

  __device__ double sum_h2(int nvec) {
    double t = 0;
    for (int i = lane; i < nvec; i += 32) t += abs2(S.h[i]);
    return warp_sum(t);
  }

  // returns false when a barrier ran out
  __device__ bool run() {
    const int c0 = (int)blockIdx.x;
    for (int i = warp; i < (a.restart ? m : a.j0); i += kCyWarps)
      for (int r = lane; r < nr; r += 32) {
        S.vr[r * ld + i] = a.vre[(long)i * n + r0 + r];
        if (C) S.vi[r * ld + i] = a.vim[(long)i * n + r0 + r];
      }
    for (int r = tid; r < nr; r += kCyThreads) {
      S.fr[r] = a.fre[r0 + r];
      if (C) S.fi[r] = a.fim[r0 + r];
    }
    if (RES) {
      const long len = (long)nr * n;
      for (long e = tid; e < len; e += kCyThreads) {
        S.ar[e] = ld_op1(a.are + r0 * n + e);
        if (C) S.ar[len + e] = ld_op1(a.aim + r0 * n + e);
      }
    }
    __syncthreads();
    double hn2 = a.st->hnorm2;
    if (a.restart) {  // V <- V Q[:, :j0], f <- (V Q)_j0 beta_hat + f sigma
      const cplx bh = a.st->beta_hat, sg = a.st->sigma;
      const int k1 = a.j0 + 1;
      for (int e = tid; e < nr * k1; e += kCyThreads) {
        const int r = e / k1, q = e - r * k1;
        double p = 0, t = 0;
        for (int i = 0; i < m; ++i) {
          const cplx z = a.Q[i + (long)q * m];
          const double v = S.vr[r * ld + i];
          p = fma(v, z.re, p);
          if (C) {
            const double u = S.vi[r * ld + i];
            p = fma(-u, z.im, p);
            t = fma(v, z.im, fma(u, z.re, t));
          }
        }
        S.xr[e] = p;
        if (C) S.xi[e] = t;
      }
      __syncthreads();
      for (int e = tid; e < nr * k1; e += kCyThreads) {
        const int q = e / nr, r = e - q * nr, x = r * k1 + q;
        const cplx v = {S.xr[x], C ? S.xi[x] : 0.0};
        if (q < a.j0) {
          S.vr[r * ld + q] = v.re;
          a.vre[(long)q * n + r0 + r] = v.re;
          if (C) {
            S.vi[r * ld + q] = v.im;
            a.vim[(long)q * n + r0 + r] = v.im;
          }
        } else {
          const cplx f = v * bh + cplx{S.fr[r], C ? S.fi[r] : 0.0} * sg;
          S.fr[r] = f.re;
          __stcg(a.fre + r0 + r, f.re);
          if (C) {
            S.fi[r] = f.im;
            __stcg(a.fim + r0 + r, f.im);
          }
        }
      }
      __syncthreads();
    }
    // after a restart on the symmetric path row j0 of H is already there
    const bool spike = a.restart && a.st->spike;
    double s2 = 0, f2;
    for (int r = tid; r < nr; r += kCyThreads) s2 += S.fr[r] * S.fr[r] + (C ? S.fi[r] * S.fi[r] : 0.0);
    norm_partial(s2);
    if (!grid_bar(a.bar, target, S.flag)) return false;
    f2 = norm2();
    int dgks = 0, brks = 0, bad = 0;
    for (int j = a.j0; j < m; ++j) {
      // invariant-subspace breakdown: a seeded random vector orthogonalised
      // against the basis, H[j][j-1] = 0
      bool brk = false;
      if (j > 0 && f2 <= 1e-24 * (hn2 + f2)) {
        brk = true;
        ++brks;
        for (int r = tid; r < nr; r += kCyThreads) {
          S.fr[r] = uniform_pm1(a.seed + j, (uint64_t)(r0 + r));
          if (C) S.fi[r] = uniform_pm1((a.seed + j) ^ 0x5851F42D4C957F2Dull, (uint64_t)(r0 + r));
        }
        __syncthreads();
        for (int sweep = 0; sweep < 2; ++sweep) {
          if (!project(S.fr, S.fi, j, S.s)) return false;
          if (!update(S.fr, S.fi, j, S.s, f2)) return false;
        }
      }
      const double beta = sqrt(f2);
      if (!(beta > 0) || isinf(beta)) {
        bad = isfinite(beta) ? 1 : 4;
        break;
      }
      const double inv = 1.0 / beta;
#pragma unroll
      for (int u = 0; u < (C ? 0 : kCyPre); ++u) {
        const int i = tid + u * kCyThreads;
        if (i < n) {
          S.xr[i] = pr[u] * inv;
        }
      }
      for (int i = tid + (C ? 0 : kCyPre) * kCyThreads; i < n; i += kCyThreads) {
        S.xr[i] = __ldcg(a.fre + i) * inv;
        if (C) S.xi[i] = __ldcg(a.fim + i) * inv;
      }
      for (int r = tid; r < nr; r += kCyThreads) {
        const double v = S.fr[r] * inv;
        S.vr[r * ld + j] = v;
        a.vre[(long)j * n + r0 + r] = v;
        if (C) {
          const double u = S.fi[r] * inv;
          S.vi[r * ld + j] = u;
          a.vim[(long)j * n + r0 + r] = u;
        }
      }
      if (c0 == 0 && tid == 0 && j > 0) {
        if (!(spike && j == a.j0))
          a.H[j + (long)(j - 1) * m] = cplx{brk ? 0.0 : beta, 0};
        else if (brk)
          for (int i = 0; i < j; ++i) a.H[j + (long)i * m] = cplx{0, 0};
      }
      __syncthreads();
      matvec();
      if (!project(S.wr, S.wi, j + 1, S.h)) return false;
      hn2 = sum_h2(j + 1);
      if (!update(S.wr, S.wi, j + 1, S.h, f2)) return false;
      if (sqrt(f2) < dgks_rho(a.rho, spike, a.j0, j) * sqrt(hn2)) {  // DGKS (ArnoldiProcedures.cpp:446-456)
        ++dgks;
        if (!project(S.fr, S.fi, j + 1, S.s)) return false;
        if (!update(S.fr, S.fi, j + 1, S.s, f2)) return false;
        if (c0 == 0)
          for (int i = tid; i <= j; i += kCyThreads) S.h[i] = S.h[i] + S.s[i];
      }
      // column j of H; its subdiagonal entry is written at the next step's
      // start (by another thread, with no barrier after this loop)
      if (c0 == 0)
        for (int i = tid; i < m; i += kCyThreads) {
          if (i == j + 1) continue;
          cplx v = i <= j ? S.h[i] : cplx{0, 0};
          if (!C) v.im = 0;
          a.H[i + (long)j * m] = v;
        }
    }
    if (c0 == 0 && tid == 0) {
      a.st->fnorm2 = f2;
      a.st->hnorm2 = hn2;
      a.st->dgks_count += dgks;
      a.st->brk_count += brks;
      a.st->status |= bad;
    }
    return true;
  }
};

template <bool C, bool RES, bool VEC>
__global__ void __launch_bounds__(kCyThreads, 1) k_arnoldi_cycle(CycleArgs a, int rows, int segs) {
  extern __shared__ __align__(16) char cy_dyn[];
  const long r0 = (long)blockIdx.x * rows;
  const int nr = (int)(r0 + rows <= a.n ? rows : (r0 < a.n ? a.n - r0 : 0));
  Cycle<C, RES, VEC> cy{a, {}, a.n, a.m, cy_ld(a.m), nr, segs, r0};
  cy_carve<C>(cy_dyn, a.n, a.m, rows, segs, RES, &cy.S);
  cy.tid = threadIdx.x;
  cy.warp = threadIdx.x >> 5;
  cy.lane = threadIdx.x & 31;
  if (!cy.run() && threadIdx.x == 0) atomicOr(&a.st->status, 2);
}

int device_limits(int* sms, int* optin) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return OAPB_ERR_CUDA;
  return OAPB_OK;
}

template <bool C, bool RES, bool VEC>
int launch(const CyclePlan& p, const CycleArgs& a, cudaStream_t s) {
  const void* k = (const void*)k_arnoldi_cycle<C, RES, VEC>;
  // (the limit is the kernel's, shared with the launches of other handles:
  // always the same)
  if (p.smem > 48 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, p.limit) != cudaSuccess)
    return OAPB_ERR_CUDA;
  CycleArgs args = a;
  int rows = p.rows, segs = p.segs;
  void* kargs[] = {&args, &rows, &segs};
  return cudaLaunchCooperativeKernel(k, dim3(p.ctas), dim3(kCyThreads), kargs, p.smem, s) == cudaSuccess
             ? OAPB_OK
             : OAPB_ERR_CUDA;
}

}  // namespace

bool cycle_plan(int n, int m, bool cplx, CyclePlan* p) {
  int sms = 0, optin = 0;
  if (m > kCyMaxM || device_limits(&sms, &optin)) return false;
  p->limit = optin;
  p->sms = sms;
  // at least eight rows per CTA: below that a CTA's share of the products is
  // shorter than what its arrival at the barriers costs
  int g = std::min(sms, (n + 7) / 8);
  if (g < 1) g = 1;
  p->rows = (n + g - 1) / g;
  p->ctas = (n + p->rows - 1) / p->rows;
  // column segments per row pair: the fewest whole rounds of the 16 warps
  const int pairs = (p->rows + 1) / 2;
  double best = 1e30;
  for (int s = 1; s <= kCyMaxSegs; ++s) {
    const double c = (double)((pairs * s + kCyWarps - 1) / kCyWarps) / s;
    if (c < best - 1e-9 && (s == 1 || n / s >= 64)) {
      best = c;
      p->segs = s;
    }
  }
  for (int res = 1; res >= 0; --res) {
    p->resident = res != 0;
    p->smem = cplx ? cy_carve<true>(nullptr, n, m, p->rows, p->segs, p->resident, nullptr)
                   : cy_carve<false>(nullptr, n, m, p->rows, p->segs, p->resident, nullptr);
    if (p->smem + 1024 <= (size_t)optin) return true;
  }
  return false;
}

int launch_cycle(const CyclePlan& p, const CycleArgs& a, cudaStream_t s) {
  const bool c = a.aim != nullptr;
  const bool vec = a.n % 2 == 0 && (((uintptr_t)a.are | (uintptr_t)a.aim) & 15) == 0;
  if (cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s) != cudaSuccess) return OAPB_ERR_CUDA;
  switch ((c ? 4 : 0) + (p.resident ? 2 : 0) + (vec ? 1 : 0)) {
    case 0: return launch<false, false, false>(p, a, s);
    case 1: return launch<false, false, true>(p, a, s);
    case 2: return launch<false, true, false>(p, a, s);
    case 3: return launch<false, true, true>(p, a, s);
    case 4: return launch<true, false, false>(p, a, s);
    case 5: return launch<true, false, true>(p, a, s);
    case 6: return launch<true, true, false>(p, a, s);
    default: return launch<true, true, true>(p, a, s);
  }
}

}  // namespace oapb
