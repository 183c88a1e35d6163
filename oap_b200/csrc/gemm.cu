// C = A B in FP64 for any sizes (CuProceduresApi::dotProduct), on the FP64
// tensor cores (mma.sync.m16n8k16.f64).
//
// The FP64 pipe bounds it: 64 multiply-adds per clock and SM, which one
// m16n8k16 instruction per warp in flight fills, while the tiles need about a
// fifth of the shared-memory bandwidth.  A CTA of 8 warps computes a BM x BN
// tile from 16-wide K chunks (cp.async, two stages, two CTAs per SM), 8 bytes
// per copy because rows of odd length are only 8-byte aligned.  Leading
// dimensions of 4 modulo 16 doubles keep the fragment reads conflict-free.
// Complex products are four real ones into two accumulators.
//
// What the sizes ask for is work for every SM: the launch takes the tile and
// the split of K with the least modelled time (gemm_plan).  The CTAs of a
// split are a cluster; they add their partial tiles through distributed shared
// memory in rank order, so the result does not depend on timing and there is
// no workspace.
//
// Complex 1500 x 1031 x 1277: 640 us (24.7 TFLOP/s of 37), 1584 us with the
// 16 x 16 FMA tile this replaces; real 1600^3: 371 us and 3118 us; complex
// 299 x 1549 x 30 (K split over clusters): 19.5 us and 99 us.
#include "gemm.cuh"

#include <algorithm>

#include "common.cuh"

namespace oapb {
namespace {

constexpr int kGmThreads = 256;
constexpr int kGmK = 16;
constexpr int kGmLda = kGmK + 4;
constexpr int kGmMaxSplit = 8;  // portable cluster size

struct GemmArgs {
  const double *are, *aim, *bre, *bim;
  double *cre, *cim;
  int M, N, K, split, tiles_m;
};

__device__ __forceinline__ void gm_cp8(uint32_t dst, const double* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0) : "memory");
}

__device__ __forceinline__ void gm_mma(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

template <int BM, int BN, bool CPLX>
struct GemmTile {
  static constexpr int kPlanes = CPLX ? 2 : 1;
  static constexpr int kLdb = BN + 4;
  static constexpr int kA = BM * kGmLda, kB = kGmK * kLdb;           // doubles of a staged plane
  static constexpr int kStage = kPlanes * (kA + kB);
  static constexpr int kWarpsN = BM == 64 && BN == 32 ? 2 : 4;       // warps across the columns
  static constexpr int kWarpsM = 8 / kWarpsN;
  static constexpr int kMT = BM / kWarpsM / 16, kNT = BN / kWarpsN / 8;  // MMA tiles of a warp
  static constexpr size_t kSmem =
      sizeof(double) * (2 * kStage > kPlanes * BM * BN ? 2 * kStage : kPlanes * BM * BN);
};

template <int BM, int BN, bool CPLX>
__global__ void __launch_bounds__(kGmThreads, 2) k_gemm(GemmArgs g) {
  using T = GemmTile<BM, BN, CPLX>;
  constexpr int P = T::kPlanes;
  extern __shared__ __align__(16) double gsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int wm = (warp / T::kWarpsN) * T::kMT * 16, wn = (warp % T::kWarpsN) * T::kNT * 8;
  const int rank = blockIdx.x % g.split;  // the cluster's CTAs are consecutive
  const unsigned tile = blockIdx.x / g.split;
  const long m0 = (long)(tile % g.tiles_m) * BM, n0 = (long)(tile / g.tiles_m) * BN;
  const double* const any = g.cre ? g.cre : g.cim;  // an address for the copies that copy nothing
  const int chunks = (g.K + kGmK - 1) / kGmK;
  const int ch0 = (int)((long)chunks * rank / g.split), ch1 = (int)((long)chunks * (rank + 1) / g.split);

  auto load = [&](int ch, int stage) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(gsm + stage * T::kStage);
    const int k0 = ch * kGmK;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const double* A = p ? g.aim : g.are;
      const double* B = p ? g.bim : g.bre;
#pragma unroll
      for (int e = tid; e < BM * kGmK; e += kGmThreads) {
        const int r = e / kGmK, c = e % kGmK;
        const bool ok = A && m0 + r < g.M && k0 + c < g.K;
        gm_cp8(base + 8u * (p * T::kA + r * kGmLda + c), ok ? A + (m0 + r) * g.K + k0 + c : any, ok);
      }
#pragma unroll
      for (int e = tid; e < BN * kGmK; e += kGmThreads) {
        const int r = e / BN, c = e % BN;
        const bool ok = B && n0 + c < g.N && k0 + r < g.K;
        gm_cp8(base + 8u * (P * T::kA + p * T::kB + r * T::kLdb + c),
               ok ? B + (long)(k0 + r) * g.N + n0 + c : any, ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double acc[P][T::kMT][T::kNT][4];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int i = 0; i < T::kMT; ++i)
#pragma unroll
      for (int j = 0; j < T::kNT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[p][i][j][e] = 0.0;

  if (ch0 < ch1) load(ch0, 0);
  for (int ch = ch0; ch < ch1; ++ch) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (ch + 1 < ch1) load(ch + 1, (ch + 1 - ch0) & 1);
    const double* As = gsm + ((ch - ch0) & 1) * T::kStage;
    const double* Bs = As + P * T::kA;
#pragma unroll
    for (int pa = 0; pa < P; ++pa) {
#pragma unroll
      for (int i = 0; i < T::kMT; ++i) {
        double a[8], na[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const double* ar = As + pa * T::kA + (wm + i * 16 + gq) * kGmLda + 4 * c + tq;
          a[2 * c] = ar[0];
          a[2 * c + 1] = ar[8 * kGmLda];
          na[2 * c] = -a[2 * c];
          na[2 * c + 1] = -a[2 * c + 1];
        }
#pragma unroll
        for (int j = 0; j < T::kNT; ++j) {
#pragma unroll
          for (int pb = 0; pb < P; ++pb) {
            double b[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) b[c] = Bs[pb * T::kB + (4 * c + tq) * T::kLdb + wn + j * 8 + gq];
            // re += re re - im im, im += re im + im re
            gm_mma(acc[CPLX ? (pa ^ pb) : 0][i][j], pa && pb ? na : a, b);
          }
        }
      }
    }
  }

  auto store = [&](int r, int c, int p, double v) {
    double* C = p ? g.cim : g.cre;
    if (C && m0 + r < g.M && n0 + c < g.N) C[(m0 + r) * g.N + n0 + c] = v;
  };
  if (g.split == 1) {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int i = 0; i < T::kMT; ++i)
#pragma unroll
        for (int j = 0; j < T::kNT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            store(wm + i * 16 + gq + (e >> 1) * 8, wn + j * 8 + 2 * tq + (e & 1), p, acc[p][i][j][e]);
  } else {
    __syncthreads();  // the staged chunks are consumed
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int i = 0; i < T::kMT; ++i)
#pragma unroll
        for (int j = 0; j < T::kNT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            gsm[p * BM * BN + (wm + i * 16 + gq + (e >> 1) * 8) * BN + wn + j * 8 + 2 * tq + (e & 1)] =
                acc[p][i][j][e];
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    // rank r adds and stores its share of the tile's elements
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(gsm);
    for (int e = rank * kGmThreads + tid; e < P * BM * BN; e += g.split * kGmThreads) {
      double v = 0;
      for (int q = 0; q < g.split; ++q) {
        uint32_t addr;
        double x;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(base + 8u * e), "r"(q));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(addr));
        v += x;
      }
      const int p = e / (BM * BN), x = e % (BM * BN);
      store(x / BN, x % BN, p, v);
    }
    // no CTA leaves while another still reads its partial tile
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  }
  if (!CPLX && g.cim)  // a real product into a complex matrix
    for (int e = rank * kGmThreads + tid; e < BM * BN; e += g.split * kGmThreads) store(e / BN, e % BN, 1, 0.0);
}

struct GemmPlan {
  int tile, split;  // tile 0: 64 x 64, 1: 64 x 32, 2: 32 x 32
};

// The tile and K split of least modelled time: rounds of CTAs over the SMs
// times a CTA's clocks (multiply-adds at 64 per clock, the smaller tiles' extra
// fragment reads as 5 and 15 %, 2000 clocks to fill and drain, 1500 for a
// split's exchange).
GemmPlan gemm_plan(int M, int N, int K, bool cplx) {
  static const int bm[3] = {64, 64, 32}, bn[3] = {64, 32, 32};
  static const double eff[3] = {1.0, 1.05, 1.15};
  const int chunks = (K + kGmK - 1) / kGmK;
  GemmPlan best{2, 1};
  double bt = 1e300;
  for (int t = 0; t < 3; ++t) {
    const double tiles = (double)((M + bm[t] - 1) / bm[t]) * ((N + bn[t] - 1) / bn[t]);
    for (int s = 1; s <= kGmMaxSplit && s <= chunks; s *= 2) {
      const double rounds = (double)(long)((tiles * s + kNumSMs - 1) / kNumSMs);
      const double chunk = (double)bm[t] * bn[t] * kGmK * (cplx ? 4 : 1) / 64.0 * eff[t];
      const double time = rounds * ((chunks + s - 1) / s) * chunk + 2000.0 + (s > 1 ? 1500.0 : 0.0);
      if (time < bt) {
        bt = time;
        best = GemmPlan{t, s};
      }
    }
  }
  return best;
}

template <int BM, int BN, bool CPLX>
int launch(GemmArgs g, cudaStream_t s) {
  using T = GemmTile<BM, BN, CPLX>;
  auto kern = k_gemm<BM, BN, CPLX>;
  if (T::kSmem > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem) != cudaSuccess)
    return OAPB_ERR_CUDA;
  g.tiles_m = (g.M + BM - 1) / BM;
  cudaLaunchConfig_t cfg = {};
  const long ctas = (long)((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN) * g.split;
  if (ctas > 0x7fffffffL) return OAPB_ERR_ARG;
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kGmThreads);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.split;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = g.split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, g) == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA;
}

template <bool CPLX>
int launch_tile(int tile, const GemmArgs& g, cudaStream_t s) {
  switch (tile) {
    case 0: return launch<64, 64, CPLX>(g, s);
    case 1: return launch<64, 32, CPLX>(g, s);
    default: return launch<32, 32, CPLX>(g, s);
  }
}

}  // namespace

int launch_gemm(const double* are, const double* aim, const double* bre, const double* bim, double* cre, double* cim,
                int M, int N, int K, cudaStream_t s) {
  const bool cplx = aim || bim || !are || !bre;
  const GemmPlan p = gemm_plan(M, N, K, cplx);
  const GemmArgs g{are, aim, bre, bim, cre, cim, M, N, K, p.split, 0};
  return cplx ? launch_tile<true>(p.tile, g, s) : launch_tile<false>(p.tile, g, s);
}

}  // namespace oapb
