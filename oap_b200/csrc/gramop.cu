// Implicit Gram operator: A v = X (X^T v) for FP32 images X (rows samples x
// cols pixels, row-major), the operator of the reference's image
// application (oap2dt3dDevice/MainAPExecutor.cpp:42-127 builds the Gram
// X X^T, or row blocks of it, on every multiplication through
// SquareMatrixApi::getDeviceMatrix / getDeviceSubMatrix,
// oapMatrixCuda/SquareMatrixApi.cpp:143-181).  Here A is never formed, and one
// application reads X once (k_gram_fused): a thread-block cluster copies a panel
// of 8 to 64 columns of all rows through shared memory into its CTAs' registers,
// forms the panel's t = X_p^T v (the CTAs' sums exchanged through distributed shared memory) and
// adds X_p t to its rows' sums, which stay in registers over all its panels.
// Above 8192 rows, beyond a cluster, and for X that is not 16-byte aligned, two
// passes over X:
//   t = X^T v   (k_gram_xt: a thread owns 4 consecutive pixels and streams a
//               slice of rows with 16-byte loads; v[r] is a broadcast; the
//               row slices' partials are summed by k_gram_reduce),
//   w = X t     (k_gram_x: one warp per row, 16-byte loads, t L2-resident).
// FP32 pixels times FP64 vectors accumulated in FP64: the result is the
// product with the exact Gram matrix of the FP32 images.
//
// For X in host memory (larger than HBM, as the reference's application
// reads its image folders block by block, MainAPExecutor.cpp:59-100,
// RecToSquareApi.cpp:71-141) the operator runs on column (pixel) blocks:
// A v = sum_c X_c (X_c^T v), so one application reads X exactly once.  The
// first blocks that fit the caller's device budget stay resident; the rest
// stream through two device buffers, the host-to-device copy of the next
// block (on its own stream) overlapping the application of the current one.
#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <tuple>

#include "common.cuh"
#include "gramop.cuh"

namespace oapb {

constexpr int kGxThreads = 256;
constexpr int kGxCols = kGxThreads * 4;  // pixels per block

__global__ void __launch_bounds__(kGxThreads) k_gram_xt(const float* __restrict__ X, int rows, int cols,
                                                       const double* __restrict__ v, int rows_per_split,
                                                       double* __restrict__ part) {
  const long c = ((long)blockIdx.x * kGxThreads + threadIdx.x) * 4;
  const int r0 = blockIdx.y * rows_per_split;
  const int r1 = min(rows, r0 + rows_per_split);
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  if (c < cols) {
    if ((cols & 3) == 0) {
      for (int r = r0; r < r1; ++r) {
        const float4 x = __ldcs(reinterpret_cast<const float4*>(X + (long)r * cols + c));
        const double vr = v[r];
        a0 = fma((double)x.x, vr, a0);
        a1 = fma((double)x.y, vr, a1);
        a2 = fma((double)x.z, vr, a2);
        a3 = fma((double)x.w, vr, a3);
      }
    } else {
      for (int r = r0; r < r1; ++r) {
        const float* xr = X + (long)r * cols;
        const double vr = v[r];
        a0 = fma((double)xr[c], vr, a0);
        if (c + 1 < cols) a1 = fma((double)xr[c + 1], vr, a1);
        if (c + 2 < cols) a2 = fma((double)xr[c + 2], vr, a2);
        if (c + 3 < cols) a3 = fma((double)xr[c + 3], vr, a3);
      }
    }
    double* p = part + (long)blockIdx.y * cols + c;
    p[0] = a0;
    if (c + 1 < cols) p[1] = a1;
    if (c + 2 < cols) p[2] = a2;
    if (c + 3 < cols) p[3] = a3;
  }
}

// t[c] = sum over the row splits (stored after the partials)
__global__ void k_gram_reduce(const double* __restrict__ part, int nsplit, int cols, double* __restrict__ t) {
  for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += (long)gridDim.x * blockDim.x) {
    double s = 0;
    for (int k = 0; k < nsplit; ++k) s += part[(long)k * cols + c];
    t[c] = s;
  }
}

__global__ void __launch_bounds__(256) k_gram_x(const float* __restrict__ X, int rows, int cols,
                                               const double* __restrict__ t, double* __restrict__ w,
                                               int accumulate) {
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * (blockDim.x >> 5);
  for (long r = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    const float* xr = X + r * cols;
    double a0 = 0, a1 = 0;
    if ((cols & 3) == 0) {
      for (int q = lane; q < cols / 4; q += 32) {
        const float4 x = __ldcs(reinterpret_cast<const float4*>(xr) + q);
        const double2 t0 = *reinterpret_cast<const double2*>(t + 4 * q);
        const double2 t1 = *reinterpret_cast<const double2*>(t + 4 * q + 2);
        a0 = fma((double)x.x, t0.x, a0);
        a1 = fma((double)x.y, t0.y, a1);
        a0 = fma((double)x.z, t1.x, a0);
        a1 = fma((double)x.w, t1.y, a1);
      }
    } else {
      for (int c = lane; c < cols; c += 32) a0 = fma((double)xr[c], t[c], a0);
    }
    const double s = warp_sum(a0 + a1);
    if (lane == 0) w[r] = accumulate ? w[r] + s : s;
  }
}

// ------------------------------------------------------- one pass over X --
// LPR lanes share a row of a panel (16 bytes each), 256 / LPR row groups; a
// thread's rows are j * groups + group (j < rpt <= 8), its part of v and its row
// sums stay in registers.  HBM should bound it: a panel's 32 KB per CTA (two
// CTAs per SM) take 1450 clocks to arrive.  FP32 -> FP64 conversion, 16 per
// clock and SM, takes 1024 when both products convert, so a panel is converted
// once into registers, which both use; the two CTAs of an SM cover one
// another's exchange of t.  Rows that are not 16-byte aligned are copied by the
// 16-byte pieces around them and read shifted (SHIFT).
// Per application, two passes against this: 4096 x 65536 460 -> 314 us, 2001 x
// 30003 195 -> 92 us, 1000 x 50000 228 -> 61 us, 660 x 41614 53 us.  Tried and
// not kept: X t a panel behind the exchange from shared memory (512 threads, one
// CTA per SM, two conversions): 275 us at 4096 rows, but 140 us at 2001 x 30003.
constexpr int kGfThreads = 256;
constexpr int kGfRows = 8;    // rows per thread
constexpr int kGfStages = 2;
constexpr int kGfMaxCluster = 8;

struct GramFusedArgs {
  const float* X;
  const double* v;
  double* part;  // clusters x rows
  int rows, cols, rpt, cluster, clusters;
  unsigned long long limit_ns;  // of every wait
  int late;  // self-test: the panel before whose sums the last CTA pauses for three limits
};

// t's exchange: each CTA writes its sums to every CTA of the cluster with
// st.async, counted by an mbarrier there.  (A cluster barrier would do, but its
// release waits for the panel copies in flight: a third of all issue slots.)
// A wait that runs out (2 s) ends the CTA with NaN sums, which the solver
// reports.  Its peers may still send it theirs, so it stays until each of them
// has left too (which they do when they have every sum, or when they miss its
// next one) and, for the sums a late peer sent last, until these have arrived or
// kGfDrainNs have passed.
constexpr unsigned long long kGfLimitNs = 2000000000ull;
constexpr unsigned long long kGfDrainNs = 1000000ull;

__device__ __forceinline__ unsigned long long gf_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool gf_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
  unsigned long long t0 = 0;
  for (unsigned it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 63u) == 63u) {
      const unsigned long long t = gf_now();
      if (!t0) t0 = t;
      if (t - t0 > limit_ns) return false;
    }
  }
}

__device__ __forceinline__ uint32_t gf_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gf_copy(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__host__ __device__ constexpr int gf_pitch(int lpr, bool shift) { return 4 * lpr + (shift ? 4 : 0); }

// FULL: every thread has kGfRows rows, all inside the matrix.  TEST: g.late holds
template <int LPR, bool SHIFT, bool FULL, bool TEST = false>
__global__ void __launch_bounds__(kGfThreads, 2) k_gram_fused(GramFusedArgs g) {
  constexpr int W = 4 * LPR, RG = kGfThreads / LPR, NW = kGfThreads / 32, P = gf_pitch(LPR, SHIFT);
  extern __shared__ __align__(16) float xs[];  // stages x (RG rpt) x P
  __shared__ __align__(16) double red[NW][W];
  __shared__ double tp[2][kGfMaxCluster][W];
  __shared__ __align__(16) double ts[W];
  __shared__ __align__(8) unsigned long long bars[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = tid % LPR, rg = tid / LPR;
  const int rank = blockIdx.x % g.cluster, cl = blockIdx.x / g.cluster;
  const int rpt = FULL ? kGfRows : g.rpt;
  const int crow = RG * rpt, r0 = rank * crow;  // the CTA's rows
  const int panels = (g.cols + W - 1) / W;
  const int iters = cl < panels ? (panels - cl + g.clusters - 1) / g.clusters : 0;
  const int stage = crow * P;
  const char* const end = reinterpret_cast<const char*>(g.X + (long)g.rows * g.cols);

  const int cstep = g.clusters * W;  // columns from one of the cluster's panels to the next
  const float* src = g.X + (long)(r0 + rg) * g.cols + (long)cl * W + 4 * q;  // this thread's piece of the next panel
  const long rstep = (long)RG * g.cols;
  const uint32_t dst0 = gf_smem(xs) + 4u * (rg * P + 4 * q);
  int lc = cl * W;  // column of the next panel to load

  auto load = [&](int i) {
    if (i < iters) {
      if (!SHIFT) {
        const uint32_t dst = dst0 + 4u * ((i % kGfStages) * stage);
        const int bytes = lc + 4 * q < g.cols ? 16 : 0;
#pragma unroll
        for (int j = 0; j < kGfRows; ++j)
          if (FULL || j < rpt) {
            const bool ok = FULL || r0 + rg + j * RG < g.rows;
            gf_copy(dst + 4u * (j * RG * P), ok && bytes ? src + j * rstep : g.X, ok ? bytes : 0);
          }
        src += cstep;
      } else {  // the LPR + 1 aligned pieces around the row's panel
        const uint32_t dst = gf_smem(xs) + 4u * ((i % kGfStages) * stage);
        for (int e = tid; e < crow * (LPR + 1); e += kGfThreads) {
          const int lr = e / (LPR + 1), ch = e - lr * (LPR + 1), r = r0 + lr;
          const char* at = reinterpret_cast<const char*>(
                               (uintptr_t)(g.X + (long)r * g.cols + lc) & ~(uintptr_t)15) + 16 * ch;
          const long left = r < g.rows ? end - at : 0;
          const int bytes = left >= 16 ? 16 : (left > 0 ? (int)left : 0);
          gf_copy(dst + 4u * (lr * P + 4 * ch), bytes ? at : (const char*)g.X, bytes);
        }
      }
      lc += cstep;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double v[kGfRows], acc[kGfRows];
#pragma unroll
  for (int j = 0; j < kGfRows; ++j) {
    const int r = r0 + j * RG + rg;
    v[j] = (FULL || (j < rpt && r < g.rows)) ? g.v[r] : 0.0;
    acc[j] = 0.0;
  }
  if (g.cluster > 1) {
    if (tid < 2) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gf_smem(&bars[tid])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // every CTA of the cluster runs, its barriers ready, before another writes there
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  }
  load(0);
  load(1);
  bool ok = true;
  int i = 0;
  for (; i < iters; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGfStages - 1) : "memory");
    if (SHIFT) __syncthreads();
    const float* x = xs + (i % kGfStages) * stage;
    double xd[kGfRows][4], s[4] = {0, 0, 0, 0};
    int valid = 4;  // columns of this lane's piece inside the matrix
    if (SHIFT) {
      const long c = ((long)cl + (long)i * g.clusters) * W + 4 * q;
      valid = g.cols - c >= 4 ? 4 : (int)(g.cols - c);
    }
#pragma unroll
    for (int j = 0; j < kGfRows; ++j) {
      if (!FULL) xd[j][0] = xd[j][1] = xd[j][2] = xd[j][3] = 0.0;
      if (FULL || j < rpt) {
        const int lr = j * RG + rg;
        if (!SHIFT) {
          const float4 f = *reinterpret_cast<const float4*>(x + lr * P + 4 * q);
          xd[j][0] = f.x;
          xd[j][1] = f.y;
          xd[j][2] = f.z;
          xd[j][3] = f.w;
        } else {
          const float* f = x + lr * P + 4 * q + (int)(((long)(r0 + lr) * g.cols) & 3);
#pragma unroll
          for (int c = 0; c < 4; ++c) xd[j][c] = c < valid ? f[c] : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) s[c] = fma(xd[j][c], v[j], s[c]);
      }
    }
    // the warp's sums over its 32 / LPR row groups: lanes that differ in bit 4
    // split the four columns, those in bit 3 the remaining two
    {
      const bool h4 = lane & 16;
      double k0 = h4 ? s[2] : s[0], k1 = h4 ? s[3] : s[1];
      const double g0 = h4 ? s[0] : s[2], g1 = h4 ? s[1] : s[3];
      if (LPR <= 16) {
        k0 += __shfl_xor_sync(0xffffffffu, g0, 16);
        k1 += __shfl_xor_sync(0xffffffffu, g1, 16);
      }
      if (LPR == 16) {
        double2* to = reinterpret_cast<double2*>(&red[warp][4 * q + (h4 ? 2 : 0)]);
        *to = make_double2(k0, k1);
      } else {
        const bool h3 = lane & 8;
        double k = h3 ? k1 : k0;
        k += __shfl_xor_sync(0xffffffffu, h3 ? k0 : k1, 8);
#pragma unroll
        for (int o = LPR; o < 8; o <<= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
        if ((lane & 7) < LPR) red[warp][4 * q + (h4 ? 2 : 0) + (h3 ? 1 : 0)] = k;
      }
    }
    __syncthreads();
    load(i + 2);  // over this panel, which is in registers
    if (tid < W) {  // the CTA's sums, to every CTA of the cluster
      double t = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) t += red[w][tid];
      if (g.cluster == 1) {
        ts[tid] = t;
      } else {
        const uint32_t at = gf_smem(&tp[i & 1][rank][tid]), bar = gf_smem(&bars[i & 1]);
        if (TEST && i == g.late && rank == g.cluster - 1)
          for (const unsigned long long t0 = gf_now(); gf_now() - t0 < 3 * g.limit_ns;) {
          }
        if (tid == 0)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"((uint32_t)(g.cluster * W * sizeof(double)))
                       : "memory");
        for (int d = 0; d < g.cluster; ++d) {
          uint32_t to, tobar;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(d));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(tobar) : "r"(bar), "r"(d));
          asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to),
                       "l"(__double_as_longlong(t)), "r"(tobar)
                       : "memory");
        }
        ok = gf_wait(bar, (i >> 1) & 1, g.limit_ns);
        t = 0;
        for (int d = 0; d < g.cluster; ++d) t += tp[i & 1][d][tid];
        ts[tid] = t;
      }
    }
    // (also the barrier after which the next iteration may overwrite red)
    if (!__syncthreads_and(ok)) {
      ok = false;
      break;
    }
    double t[4];
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
      const double2 u = *reinterpret_cast<const double2*>(&ts[4 * q + c]);
      t[c] = u.x;
      t[c + 1] = u.y;
    }
#pragma unroll
    for (int j = 0; j < kGfRows; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j] = fma(xd[j][c], t[c], acc[j]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (!ok) {  // (only with a cluster)
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    gf_wait(gf_smem(&bars[i & 1]), (i >> 1) & 1, kGfDrainNs);
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kGfRows; ++j)
    if (FULL || j < rpt) {
      const int r = r0 + j * RG + rg;
      double a = acc[j];
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (q == 0 && r < g.rows) g.part[(long)cl * g.rows + r] = ok ? a : __longlong_as_double(0x7ff8000000000000ll);
    }
}

// w[r] = (accumulate: w[r] +) sum over the clusters: a block owns 32 rows, its
// 8 warps every eighth cluster, added in a fixed order
__global__ void __launch_bounds__(256) k_gram_rows(const double* __restrict__ part, int clusters, int rows,
                                                   double* __restrict__ w, int accumulate) {
  __shared__ double red[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * 32 + lane;
  double s = 0;
  if (r < rows)
    for (int c = warp; c < clusters; c += 8) s += part[(long)c * rows + r];
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && r < rows) {
    double t = accumulate ? w[r] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) t += red[u][lane];
    w[r] = t;
  }
}

struct GramFusedPlan {
  int lpr = 0, cluster = 1, rpt = 1;
};
// the widest panel whose rows fit the cluster's threads; false above 8192 rows
static bool gram_fused_plan(int rows, GramFusedPlan* p) {
  const int one = kGfThreads * kGfRows;  // rows x LPR of a CTA
  p->lpr = rows <= one / 16 ? 16 : rows <= one / 8 ? 8 : rows <= kGfMaxCluster * (one / 4) ? 4 : 2;
  const int cap = one / p->lpr;
  p->cluster = (rows + cap - 1) / cap;
  if (p->cluster > kGfMaxCluster) return false;
  const int rg = kGfThreads / p->lpr * p->cluster;
  p->rpt = (rows + rg - 1) / rg;
  return true;
}

static cudaLaunchConfig_t gram_config(const GramFusedPlan& p, int clusters, size_t smem, cudaStream_t s,
                                      cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * p.cluster));
  cfg.blockDim = dim3(kGfThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)p.cluster;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

constexpr int kGfMaxClusters = 2 * kNumSMs;

// clusters that run at once, asked once per device and shape
template <typename K>
static int max_clusters(K kern, const GramFusedPlan& p, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, size_t>, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  const auto key = std::make_tuple(dev, (const void*)kern, p.cluster, smem);
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = gram_config(p, 1, smem, nullptr, &at);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = std::max(1, kNumSMs / p.cluster);
  }
  n = std::min(n, kGfMaxClusters);
  known[key] = n;
  return n;
}

template <int LPR, bool SHIFT, bool FULL>
static int gram_fused(const GramFusedPlan& p, GramFusedArgs g, double* w, bool accumulate, cudaStream_t s) {
  auto kern = k_gram_fused<LPR, SHIFT, FULL>;
  constexpr size_t row_group = sizeof(float) * kGfStages * (kGfThreads / LPR) * gf_pitch(LPR, SHIFT);
  const size_t smem = row_group * p.rpt;
  // the limit is the kernel's, shared with every other thread's launches: always
  // what the most rows per thread take
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(row_group * kGfRows)) !=
      cudaSuccess)
    return OAPB_ERR_CUDA;
  g.clusters = std::min(max_clusters(kern, p, smem), (g.cols + 4 * LPR - 1) / (4 * LPR));
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = gram_config(p, g.clusters, smem, s, &at);
  if (cudaLaunchKernelEx(&cfg, kern, g) != cudaSuccess) return OAPB_ERR_CUDA;
  k_gram_rows<<<(g.rows + 31) / 32, 256, 0, s>>>(g.part, g.clusters, g.rows, w, accumulate ? 1 : 0);
  return cudaGetLastError() == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA;
}

template <int LPR>
static int gram_fused_any(const GramFusedPlan& p, const GramFusedArgs& g, double* w, bool accumulate, cudaStream_t s) {
  const bool full = p.rpt == kGfRows && g.rows == kGfThreads / LPR * kGfRows * p.cluster;
  if (g.cols & 3)
    return full ? gram_fused<LPR, true, true>(p, g, w, accumulate, s)
                : gram_fused<LPR, true, false>(p, g, w, accumulate, s);
  return full ? gram_fused<LPR, false, true>(p, g, w, accumulate, s)
              : gram_fused<LPR, false, false>(p, g, w, accumulate, s);
}

static int gram_op_splits(int rows, int cols) {
  const int tiles = (cols + kGxCols - 1) / kGxCols;
  int s = (4 * kNumSMs + tiles - 1) / tiles;
  if (s > 64) s = 64;
  if (s > rows) s = rows;
  return s < 1 ? 1 : s;
}

size_t gram_op_workspace(int rows, int cols) {
  GramFusedPlan p;
  const size_t two = ((size_t)gram_op_splits(rows, cols) + 1) * cols;
  return gram_fused_plan(rows, &p) ? std::max(two, (size_t)kGfMaxClusters * rows) : two;
}

int launch_gram_apply(const float* X, int rows, int cols, const double* v, double* w, double* ws, cudaStream_t s,
                      bool accumulate) {
  if (!X || !v || !w || !ws || rows < 1 || cols < 1) return OAPB_ERR_ARG;
  if ((cols & 3) == 0 && ((uintptr_t)X & 15)) return OAPB_ERR_ARG;
  GramFusedPlan p;
  if (((uintptr_t)X & 15) == 0 && gram_fused_plan(rows, &p)) {
    const GramFusedArgs g{X, v, ws, rows, cols, p.rpt, p.cluster, 0, kGfLimitNs, -1};
    switch (p.lpr) {
      case 16: return gram_fused_any<16>(p, g, w, accumulate, s);
      case 8: return gram_fused_any<8>(p, g, w, accumulate, s);
      case 4: return gram_fused_any<4>(p, g, w, accumulate, s);
      default: return gram_fused_any<2>(p, g, w, accumulate, s);
    }
  }
  const int ns = gram_op_splits(rows, cols);
  const int rps = (rows + ns - 1) / ns;
  double* t = ws + (size_t)ns * cols;
  k_gram_xt<<<dim3((cols + kGxCols - 1) / kGxCols, ns), kGxThreads, 0, s>>>(X, rows, cols, v, rps, ws);
  k_gram_reduce<<<grid_for(cols, 256, kNumSMs * 4), 256, 0, s>>>(ws, ns, cols, t);
  k_gram_x<<<grid_for((long)rows * 32, 256, kNumSMs * 8), 256, 0, s>>>(X, rows, cols, t, w, accumulate ? 1 : 0);
  return cudaGetLastError() == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA;
}

// ------------------------------------------------------------ host X --
struct GramStream {
  const float* hX = nullptr;  // host, rows x cols row-major
  int rows = 0, cols = 0, bc = 0, nb = 0, resident = 0;
  float* dres = nullptr;      // resident blocks, each rows x bc (the last may be narrower)
  float* dbuf[2] = {nullptr, nullptr};
  double* ws = nullptr;       // gram_op_workspace(rows, bc)
  cudaStream_t cs = nullptr;  // copy stream
  cudaEvent_t copied[2] = {nullptr, nullptr}, consumed[2] = {nullptr, nullptr};
  unsigned long long streamed_bytes = 0;
};

static int block_width(const GramStream* g, int c) { return std::min(g->bc, g->cols - c * g->bc); }

void gram_stream_destroy(GramStream* g) {
  if (!g) return;
  if (g->cs) cudaStreamSynchronize(g->cs);
  for (int i = 0; i < 2; ++i) {
    if (g->dbuf[i]) cudaFree(g->dbuf[i]);
    if (g->copied[i]) cudaEventDestroy(g->copied[i]);
    if (g->consumed[i]) cudaEventDestroy(g->consumed[i]);
  }
  if (g->dres) cudaFree(g->dres);
  if (g->ws) cudaFree(g->ws);
  if (g->cs) cudaStreamDestroy(g->cs);
  delete g;
}

int gram_stream_create(const float* hX, int rows, int cols, int block_cols, unsigned long long resident_bytes,
                       cudaStream_t s, GramStream** out) {
  if (!hX || rows < 1 || cols < 1 || block_cols < 1 || !out) return OAPB_ERR_ARG;
  GramStream* g = new (std::nothrow) GramStream();
  if (!g) return OAPB_ERR_NOMEM;
  g->hX = hX;
  g->rows = rows;
  g->cols = cols;
  g->bc = std::min(cols, (block_cols + 3) / 4 * 4);  // 16-byte rows for the vector loads
  g->nb = (cols + g->bc - 1) / g->bc;
  const size_t block_bytes = sizeof(float) * (size_t)rows * g->bc;
  g->resident = (int)std::min<unsigned long long>((unsigned long long)g->nb, resident_bytes / block_bytes);
  int rc = OAPB_OK;
  do {
    if (cudaMalloc(&g->ws, sizeof(double) * gram_op_workspace(rows, g->bc)) != cudaSuccess) {
      rc = OAPB_ERR_NOMEM;
      break;
    }
    if (g->resident > 0 && cudaMalloc(&g->dres, block_bytes * g->resident) != cudaSuccess) {
      rc = OAPB_ERR_NOMEM;
      break;
    }
    if (g->resident < g->nb) {
      for (int i = 0; i < 2 && !rc; ++i) {
        if (cudaMalloc(&g->dbuf[i], block_bytes) != cudaSuccess) rc = OAPB_ERR_NOMEM;
        else if (cudaEventCreateWithFlags(&g->copied[i], cudaEventDisableTiming) != cudaSuccess ||
                 cudaEventCreateWithFlags(&g->consumed[i], cudaEventDisableTiming) != cudaSuccess)
          rc = OAPB_ERR_CUDA;
      }
      if (!rc && cudaStreamCreateWithFlags(&g->cs, cudaStreamNonBlocking) != cudaSuccess) rc = OAPB_ERR_CUDA;
      if (rc) break;
    }
    // the resident blocks, copied once
    for (int c = 0; c < g->resident; ++c) {
      const int w = block_width(g, c);
      if (cudaMemcpy2DAsync(g->dres + (size_t)c * rows * g->bc, sizeof(float) * w, hX + (size_t)c * g->bc,
                            sizeof(float) * cols, sizeof(float) * w, rows, cudaMemcpyHostToDevice, s) !=
          cudaSuccess) {
        rc = OAPB_ERR_CUDA;
        break;
      }
    }
  } while (0);
  if (rc) {
    cudaGetLastError();
    gram_stream_destroy(g);
    return rc;
  }
  *out = g;
  return OAPB_OK;
}

int gram_stream_apply(GramStream* g, const double* v, double* w, cudaStream_t s) {
  int slot = 0;
  for (int c = 0; c < g->nb; ++c) {
    const int wc = block_width(g, c);
    const float* Xc;
    bool streamed = c >= g->resident;
    if (!streamed) {
      Xc = g->dres + (size_t)c * g->rows * g->bc;
    } else {
      // the slot's previous block has been read; then copy this block into it
      if (cudaStreamWaitEvent(g->cs, g->consumed[slot], 0) != cudaSuccess ||
          cudaMemcpy2DAsync(g->dbuf[slot], sizeof(float) * wc, g->hX + (size_t)c * g->bc, sizeof(float) * g->cols,
                            sizeof(float) * wc, g->rows, cudaMemcpyHostToDevice, g->cs) != cudaSuccess ||
          cudaEventRecord(g->copied[slot], g->cs) != cudaSuccess ||
          cudaStreamWaitEvent(s, g->copied[slot], 0) != cudaSuccess)
        return OAPB_ERR_CUDA;
      g->streamed_bytes += sizeof(float) * (unsigned long long)wc * g->rows;
      Xc = g->dbuf[slot];
    }
    const int rc = launch_gram_apply(Xc, g->rows, wc, v, w, g->ws, s, c > 0);
    if (rc) return rc;
    if (streamed) {
      if (cudaEventRecord(g->consumed[slot], s) != cudaSuccess) return OAPB_ERR_CUDA;
      slot ^= 1;
    }
  }
  return OAPB_OK;
}

unsigned long long gram_stream_bytes(const GramStream* g) { return g ? g->streamed_bytes : 0; }
int gram_stream_resident_blocks(const GramStream* g) { return g ? g->resident : 0; }
int gram_stream_blocks(const GramStream* g) { return g ? g->nb : 0; }

}  // namespace oapb

using namespace oapb;

extern "C" int oapb_selftest_gram_wait(uint32_t limit_us, int32_t late, int32_t* timed_out, void* stream) {
  constexpr int kRows = 4096, kCols = 256;  // one cluster of 8 CTAs, 16 panels of 16 columns
  if (!timed_out || limit_us == 0 || limit_us > 100000u || late < -1 || late >= kCols / 16) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  GramFusedPlan p;
  if (!gram_fused_plan(kRows, &p) || p.lpr != 4 || p.rpt != kGfRows) return OAPB_ERR_ARG;
  auto kern = k_gram_fused<4, false, true, true>;
  const size_t smem = sizeof(float) * kGfStages * (kGfThreads / 4) * kGfRows * gf_pitch(4, false);
  const size_t xb = sizeof(float) * kRows * kCols, vb = sizeof(double) * kRows;
  char* buf = nullptr;
  if (cudaMallocAsync((void**)&buf, xb + 2 * vb, s) != cudaSuccess) return OAPB_ERR_NOMEM;
  static double part[kRows];
  static std::mutex mu;  // of part
  std::lock_guard<std::mutex> lock(mu);
  const GramFusedArgs g{(const float*)buf, (const double*)(buf + xb), (double*)(buf + xb + vb),
                        kRows, kCols, p.rpt, p.cluster, 1, (unsigned long long)limit_us * 1000ull, late};
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = gram_config(p, 1, smem, s, &at);
  int rc = OAPB_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaMemsetAsync(buf, 0, xb + 2 * vb, s) != cudaSuccess || cudaLaunchKernelEx(&cfg, kern, g) != cudaSuccess ||
      cudaMemcpyAsync(part, g.part, vb, cudaMemcpyDeviceToHost, s) != cudaSuccess)
    rc = OAPB_ERR_CUDA;
  cudaFreeAsync(buf, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) rc = OAPB_ERR_CUDA;
  if (rc) return rc;
  *timed_out = 0;
  for (double x : part) *timed_out |= x != x;
  return *timed_out ? OAPB_ERR_TIMEOUT : OAPB_OK;
}
