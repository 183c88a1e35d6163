// Warm-start network and parametric operators.
//
// 1. oapb_param_operators: A(theta_p) = A0 + sum_i theta_p[i] B_i for a batch
//    of parameter vectors (each basis element read once, written P times).
// 2. A dense MLP with BF16 weights and activations and FP32 accumulation:
//    forward, backward (data and weight gradients) and an Adam step on FP32
//    master weights, all on the device.  Each layer's outputs pass through
//    one of the reference's activations (oapNeuralHost/oapLayerStructure.h:
//    32-38, applied by activateFunc / derivativeFunc,
//    oapGenericNeuralApi.h:43-120): LINEAR, SIGMOID, TANH or SIN; by
//    default tanh hidden layers and a linear output.
//    The network maps an operator's parameters theta to a warm-start vector
//    and a shift set for the Arnoldi method.  Nearest reference analogue:
//    the generic forward / back-propagation of the neural library
//    (oapNeuralHost/oapGenericNeuralApi.h:195-360) over CuProceduresApi ops
//    (dotProduct, tensorProduct, sum).
//
// Every layer product is one kernel, k_layer: C[M x N] = sum_k A(m, k) B(n, k)
// with BF16 operands contiguous in either index (the forward product, the data
// gradient and the weight gradient differ only in that), FP32 accumulation and
// the layer's elementwise work as its epilogue (bias and activation; the
// activation's derivative; the bias gradient beside the weight gradient).
//
// The sums run in k order on the FP32 pipe, not on the tensor cores: every
// product rounds its result to BF16 for the next one, and another summation
// order moves some of those roundings to the other neighbour, which training
// then amplifies (a tensor-core version took 139 us per step, but two steps
// moved the gradients by 1e-3 of their norm; this one gives the bits of the
// 32 x 32 tile it replaces).  The network is small (a step of
// 16 - 256 - 256 - 2056 on 256 samples is 0.9 GFLOP), so what bounds it is the
// chain of launches and the longest K loop: 16-byte loads of rows padded to 8
// values, operands staged as FP32 once, two stages with the next chunk's loads
// in flight, smaller tiles where a product has few, launches that overlap
// their predecessors.
#include <cuda_bf16.h>
#include <math.h>

#include <new>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "matio.cuh"
#include "streamk.cuh"

namespace oapb {

// ------------------------------------------------------ parametric operator
__global__ void k_param_operators(const double* __restrict__ A0, const double* const* __restrict__ Bs, int nparams,
                                  const double* __restrict__ theta, int P, long nn, double* __restrict__ out) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < nn; e += (long)gridDim.x * blockDim.x) {
    double base = A0[e];
    double b[32];
    for (int i = 0; i < nparams; ++i) b[i] = Bs[i][e];
    for (int p = 0; p < P; ++p) {
      double v = base;
      for (int i = 0; i < nparams; ++i) v += theta[(long)p * nparams + i] * b[i];
      out[(long)p * nn + e] = v;
    }
  }
}

// ------------------------------------------------------------ layer GEMM --
constexpr int kLK = 32;         // k chunk
constexpr int kLThreads = 256;  // 16 x 16
constexpr int kBiasBatch = 32;

__host__ __device__ inline int pad8(int x) { return (x + 7) & ~7; }

// activation of a layer's outputs (oapb_activation) and its derivative from
// the pre-activation z and the output h
__device__ __forceinline__ float act_f(float z, int act) {
  switch (act) {
    case OAPB_ACT_SIGMOID: return 1.f / (1.f + expf(-z));
    case OAPB_ACT_TANH: return tanhf(z);
    case OAPB_ACT_SIN: return sinf(z);
    default: return z;
  }
}
__device__ __forceinline__ float act_df(float z, float h, int act) {
  switch (act) {
    case OAPB_ACT_SIGMOID: return h * (1.f - h);
    case OAPB_ACT_TANH: return 1.f - h * h;
    case OAPB_ACT_SIN: return cosf(z);
    default: return 1.f;
  }
}

// Operand X(r, k) of a product: X[r * ld + k] (K-contiguous) or X[k * ld + r];
// ld a multiple of 8, the pad of a row zero.
struct LayerArgs {
  const __nv_bfloat16 *A, *B;
  int lda, ldb;
  int M, N, K, tiles_n, tiles;
  // outputs, each may be null: C FP32 and Z FP32 (ldc = N), Cb BF16 (ldcb)
  float* C;
  float* Z;
  __nv_bfloat16* Cb;
  int ldcb;
  const float* bias;     // mode 1
  const float *H, *Zin;  // mode 2: outputs and pre-activations of the layer below
  int act;
  const float* dZ;       // mode 0: FP32 K x M, its column sums to db
  float* db;
};

// 8 values (16 bytes) of a staged chunk: rows r .. of one k (row-contiguous) or
// k .. of one row, zero outside the operand
template <int ROWS, bool KC>
struct LayerStage {
  static constexpr int kCopies = ROWS * kLK / 8;
  // copy e of the chunk: (row, k) of its first value
  __device__ static __forceinline__ void at(int e, int& r, int& k) {
    if (KC) {
      r = e % ROWS;
      k = e / ROWS * 8;
    } else {
      r = e % (ROWS / 8) * 8;
      k = e / (ROWS / 8);
    }
  }
  __device__ static __forceinline__ uint4 load(const __nv_bfloat16* X, int ld, int r0, int rows, int k0, int K, int e) {
    int r, k;
    at(e, r, k);
    r += r0;
    k += k0;
    if (r >= rows || k >= K) return make_uint4(0, 0, 0, 0);
    return *reinterpret_cast<const uint4*>(KC ? X + (long)r * ld + k : X + (long)k * ld + r);
  }
  // as FP32 into s[k][ROWS]
  __device__ static __forceinline__ void put(float* s, int e, const uint4& v) {
    int r, k;
    at(e, r, k);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float f[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
    if (KC) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s[(k + i) * ROWS + r] = f[i];
    } else {
      *reinterpret_cast<float4*>(s + k * ROWS + r) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(s + k * ROWS + r + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
  }
};

// db[n] = sum_b dZ[b][n] in order of b, one thread per column
__device__ __forceinline__ void bias_grad(const float* __restrict__ dZ, int B, int N, int n, float* db) {
  if (n >= N) return;
  float s = 0;
  for (int b0 = 0; b0 < B; b0 += kBiasBatch) {
    float v[kBiasBatch];
#pragma unroll
    for (int u = 0; u < kBiasBatch; ++u) v[u] = b0 + u < B ? dZ[(long)(b0 + u) * N + n] : 0.f;
#pragma unroll
    for (int u = 0; u < kBiasBatch; ++u)
      if (b0 + u < B) s += v[u];
  }
  db[n] = s;
}

// MODE 0: C, and the column sums of dZ on the blocks past the tiles; 1: z = C +
// bias (kept in Z when given), act(z); 2: C act'(h).  A thread computes TM / 16
// x 2 outputs of a TM x 32 tile.
template <int MODE, bool AK, bool BK, int TM>
__global__ void __launch_bounds__(kLThreads) k_layer(LayerArgs g) {
  constexpr int TN = 32, RM = TM / 16;
  using SA = LayerStage<TM, AK>;
  using SB = LayerStage<TN, BK>;
  static_assert(SA::kCopies + SB::kCopies <= kLThreads, "one copy per thread");
  __shared__ __align__(16) float As[2][kLK * TM];
  __shared__ __align__(16) float Bs[2][kLK * TN];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  if (MODE == 0 && (int)blockIdx.x >= g.tiles) {
    bias_grad(g.dZ, g.K, g.M, ((int)blockIdx.x - g.tiles) * kLThreads + tid, g.db);
    return;
  }
  const int n0 = (blockIdx.x % g.tiles_n) * TN, m0 = (blockIdx.x / g.tiles_n) * TM;
  const int chunks = (g.K + kLK - 1) / kLK;
  const bool ld_a = tid < SA::kCopies, ld_b = !ld_a && tid - SA::kCopies < SB::kCopies;
  auto load = [&](int c) {
    return ld_a ? SA::load(g.A, g.lda, m0, g.M, c * kLK, g.K, tid)
                : ld_b ? SB::load(g.B, g.ldb, n0, g.N, c * kLK, g.K, tid - SA::kCopies) : make_uint4(0, 0, 0, 0);
  };
  auto put = [&](int st, const uint4& v) {
    if (ld_a) SA::put(As[st], tid, v);
    if (ld_b) SB::put(Bs[st], tid - SA::kCopies, v);
  };
  float acc[RM][2] = {};
  put(0, load(0));
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    const bool more = c + 1 < chunks;
    uint4 nx = make_uint4(0, 0, 0, 0);
    if (more) nx = load(c + 1);
    const float *a = As[c & 1] + ty * RM, *b = Bs[c & 1] + 2 * tx;
#pragma unroll
    for (int k = 0; k < kLK; ++k) {
      float av[RM];
      if (RM == 2) {
        const float2 t = *reinterpret_cast<const float2*>(a + k * TM);
        av[0] = t.x;
        av[RM - 1] = t.y;
      } else {
        av[0] = a[k * TM];
      }
      const float2 bv = *reinterpret_cast<const float2*>(b + k * TN);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        acc[i][0] = fmaf(av[i], bv.x, acc[i][0]);
        acc[i][1] = fmaf(av[i], bv.y, acc[i][1]);
      }
    }
    if (more) put((c + 1) & 1, nx);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int m = m0 + ty * RM + i, n = n0 + tx * 2 + j;
      if (m >= g.M) continue;
      if (n >= g.N) {  // the BF16 row's pad
        if (g.Cb && n < g.ldcb) g.Cb[(long)m * g.ldcb + n] = __float2bfloat16_rn(0.f);
        continue;
      }
      const long at = (long)m * g.N + n;
      float v = acc[i][j];
      if (MODE == 1) {
        v += g.bias[n];
        if (g.Z) g.Z[at] = v;
        v = act_f(v, g.act);
      } else if (MODE == 2) {
        v *= act_df(g.Zin ? g.Zin[at] : 0.f, g.H[at], g.act);
      }
      if (g.C) g.C[at] = v;
      if (g.Cb) g.Cb[(long)m * g.ldcb + n] = __float2bfloat16_rn(v);
    }
}

// Output layer: dZ = (Y - T) / B times the activation's derivative (FP32, and
// BF16 with row length ldb), and the loss sum (y - t)^2 / (2 B), one atomic per
// block
__global__ void __launch_bounds__(256) k_out_grad(const float* __restrict__ Y, const float* __restrict__ T,
                                                 const float* __restrict__ Z, int act, int B, int N,
                                                 __nv_bfloat16* dZb, int ldb, float* dZf, double* loss) {
  __shared__ double red[8];
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  double s = 0;
  const long len = (long)B * ldb;
  for (long x = (long)blockIdx.x * blockDim.x + threadIdx.x; x < len; x += (long)gridDim.x * blockDim.x) {
    const long b = x / ldb;
    const int n = (int)(x - b * ldb);
    if (n >= N) {  // the rows' pad
      dZb[x] = __float2bfloat16_rn(0.f);
      continue;
    }
    const long e = b * N + n;
    const float y = Y[e], d = y - T[e];
    s += (double)d * d;
    float g = d / (float)B;
    if (act != OAPB_ACT_LINEAR) g *= act_df(Z ? Z[e] : 0.f, y, act);
    dZb[x] = __float2bfloat16_rn(g);
    dZf[e] = g;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double q = 0;
    for (int w = 0; w < 8; ++w) q += red[w];
    atomicAdd(loss, 0.5 * q / B);
  }
}

// where the layers' weights lie: FP32 masters packed, BF16 copies with padded rows
struct WeightMap {
  int nl;
  long off[9];    // first master of layer l; off[nl] = all weights
  long boff[8];   // first BF16 value of layer l
  int in[8];      // row length
};
__device__ __forceinline__ long weight_bf16_index(const WeightMap& m, long e) {
  int l = 0;
  while (l + 1 < m.nl && e >= m.off[l + 1]) ++l;
  const long r = e - m.off[l];
  const int in = m.in[l];
  return m.boff[l] + (r / in) * pad8(in) + r % in;
}

// Adam on FP32 masters; BF16 working copy refreshed
__global__ void k_adam(float* w, const float* g, float* m1, float* m2, long len, float lr, float b1, float b2,
                       float eps, float c1, float c2, __nv_bfloat16* wb, WeightMap map) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // dependent launch
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < len; e += (long)gridDim.x * blockDim.x) {
    const float gg = g[e];
    const float a = b1 * m1[e] + (1.f - b1) * gg;
    const float v = b2 * m2[e] + (1.f - b2) * gg * gg;
    m1[e] = a;
    m2[e] = v;
    const float nw = w[e] - lr * (a / c1) / (sqrtf(v / c2) + eps);
    w[e] = nw;
    if (e < map.off[map.nl]) wb[weight_bf16_index(map, e)] = __float2bfloat16_rn(nw);
  }
}

// the BF16 copies of all weights
__global__ void k_weights_bf16(const float* w, __nv_bfloat16* wb, WeightMap map) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < map.off[map.nl]; e += (long)gridDim.x * blockDim.x)
    wb[weight_bf16_index(map, e)] = __float2bfloat16_rn(w[e]);
}

// rows of n values to BF16 rows of ld
__global__ void k_rows_bf16(const float* __restrict__ x, int n, long len, int ld, __nv_bfloat16* y) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < len; e += (long)gridDim.x * blockDim.x)
    y[(e / n) * ld + e % n] = __float2bfloat16_rn(x[e]);
}

__global__ void k_init_uniform(float* w, long len, float scale, uint64_t seed) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < len; e += (long)gridDim.x * blockDim.x)
    w[e] = (float)(scale * uniform_pm1(seed, (uint64_t)e));
}

}  // namespace oapb

using namespace oapb;

struct oapb_mlp {
  int nl = 0;                 // layers
  std::vector<int> sz;        // nl + 1 sizes
  std::vector<long> woff, boff;
  long nparam = 0;
  float *w = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;  // FP32 [all weights | all biases]
  __nv_bfloat16* wb = nullptr;                                     // BF16 copies of the weights (rows padded)
  WeightMap map{};
  int step = 0;
  std::vector<int> act;                // activation of each layer's outputs (oapb_activation)
  // activations for the last forward (capacity batch)
  int cap = 0;
  void* acts = nullptr;                // the buffers below
  std::vector<float*> hf;              // FP32 activations per layer output (nl)
  std::vector<float*> zf;              // FP32 pre-activations per layer output (nl)
  std::vector<__nv_bfloat16*> hb;      // BF16 activations: input + per layer (rows padded)
  float* dA[2] = {nullptr, nullptr};   // FP32 dZ of two layers in turn (cap x max size)
  __nv_bfloat16* dAb[2] = {nullptr, nullptr};  // BF16, rows padded
  double* loss = nullptr;
};

namespace {

void free_acts(oapb_mlp* h) {
  if (h->acts) cudaFree(h->acts);
  h->acts = nullptr;
  h->cap = 0;
}

// The buffers of a batch, one allocation, zeroed: the row pads stay zero.
// (Fourteen allocations with a fill each took most of a new network's first
// step: 16 - 256 - 256 - 2056 at 256 samples 2.3 ms, 0.6 with one.)
int ensure_acts(oapb_mlp* h, int batch, cudaStream_t s) {
  if (batch <= h->cap) return OAPB_OK;
  free_acts(h);
  int mx = 0;
  for (int v : h->sz) mx = v > mx ? v : mx;
  h->hb.assign(h->nl + 1, nullptr);
  h->hf.assign(h->nl, nullptr);
  h->zf.assign(h->nl, nullptr);
  char* base = nullptr;
  size_t total = 0;
  for (int pass = 0; pass < 2; ++pass) {  // sizes, then addresses
    size_t off = 0;
    auto take = [&](auto** p, size_t values) {
      if (base) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(base + off);
      off += (values * sizeof(**p) + 255) & ~(size_t)255;
    };
    const size_t b = (size_t)batch;
    for (int l = 0; l <= h->nl; ++l) take(&h->hb[l], b * pad8(h->sz[l]));
    for (int l = 0; l < h->nl; ++l) {
      take(&h->hf[l], b * h->sz[l + 1]);
      take(&h->zf[l], b * h->sz[l + 1]);
    }
    for (int i = 0; i < 2; ++i) {
      take(&h->dA[i], b * mx);
      take(&h->dAb[i], b * pad8(mx));
    }
    if (pass == 0) {
      total = off;
      if (cudaMalloc(&h->acts, total) != cudaSuccess) {
        h->acts = nullptr;
        cudaGetLastError();
        return OAPB_ERR_NOMEM;
      }
      base = (char*)h->acts;
    }
  }
  if (cudaMemsetAsync(h->acts, 0, total, s) != cudaSuccess) return OAPB_ERR_CUDA;
  h->cap = batch;
  return OAPB_OK;
}

template <int MODE, bool AK, bool BK>
int layer(LayerArgs g, cudaStream_t s) {
  // 32 x 32 tiles, 16 x 32 where those leave SMs idle
  const int tn = (g.N + 31) / 32, tall = tn * ((g.M + 31) / 32);
  const int tm = tall >= kNumSMs ? 32 : 16;
  g.tiles_n = tn;
  g.tiles = tn * ((g.M + tm - 1) / tm);
  const int extra = MODE == 0 ? (g.M + kLThreads - 1) / kLThreads : 0;
  const cudaError_t e =
      tm == 32 ? launch_dependent(k_layer<MODE, AK, BK, 32>, dim3(g.tiles + extra), dim3(kLThreads), 0, s, g)
               : launch_dependent(k_layer<MODE, AK, BK, 16>, dim3(g.tiles + extra), dim3(kLThreads), 0, s, g);
  return e == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA;
}

int forward_impl(oapb_mlp* h, const float* x, int B, cudaStream_t s) {
  int rc = ensure_acts(h, B, s);
  if (rc) return rc;
  const long n0 = (long)B * h->sz[0];
  k_rows_bf16<<<grid_for(n0, 256), 256, 0, s>>>(x, h->sz[0], n0, pad8(h->sz[0]), h->hb[0]);
  for (int l = 0; l < h->nl && !rc; ++l) {
    const int in = h->sz[l], out = h->sz[l + 1];
    LayerArgs g{};
    g.A = h->hb[l];
    g.B = h->wb + h->map.boff[l];
    g.lda = g.ldb = pad8(in);
    g.M = B;
    g.N = out;
    g.K = in;
    g.C = h->hf[l];
    g.Z = h->act[l] == OAPB_ACT_SIN ? h->zf[l] : nullptr;
    g.Cb = h->hb[l + 1];
    g.ldcb = pad8(out);
    g.bias = h->w + h->boff[l];
    g.act = h->act[l];
    rc = layer<1, true, true>(g, s);
  }
  return rc ? rc : (cudaGetLastError() == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA);
}

}  // namespace

extern "C" {

int oapb_param_operators(const double* A0, const double* const* B, uint32_t nparams, const double* theta,
                         uint32_t count, uint32_t n, double* out, void* stream) {
  if (!A0 || !B || !theta || !out || nparams == 0 || nparams > 32 || count == 0 || n == 0) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const double** dB = nullptr;
  if (cudaMallocAsync((void**)&dB, sizeof(double*) * nparams, s) != cudaSuccess) return OAPB_ERR_NOMEM;
  int rc = OAPB_OK;
  if (cudaMemcpyAsync(dB, B, sizeof(double*) * nparams, cudaMemcpyHostToDevice, s) != cudaSuccess) rc = OAPB_ERR_CUDA;
  if (!rc) {
    const long nn = (long)n * n;
    k_param_operators<<<grid_for(nn, 256, kNumSMs * 8), 256, 0, s>>>(A0, dB, (int)nparams, theta, (int)count, nn,
                                                                      out);
    if (cudaGetLastError() != cudaSuccess) rc = OAPB_ERR_CUDA;
  }
  cudaFreeAsync(dB, s);
  return rc;
}

int oapb_mlp_create(oapb_mlp** out, const uint32_t* sizes, uint32_t nlayers, uint64_t seed) {
  if (!out || !sizes || nlayers < 1 || nlayers > 8) return OAPB_ERR_ARG;
  oapb_mlp* h = new (std::nothrow) oapb_mlp();
  if (!h) return OAPB_ERR_NOMEM;
  h->nl = (int)nlayers;
  for (uint32_t i = 0; i <= nlayers; ++i) {
    if (sizes[i] == 0) {
      delete h;
      return OAPB_ERR_ARG;
    }
    h->sz.push_back((int)sizes[i]);
  }
  long off = 0;
  for (int l = 0; l < h->nl; ++l) {
    h->woff.push_back(off);
    off += (long)h->sz[l] * h->sz[l + 1];
  }
  const long nw = off;
  for (int l = 0; l < h->nl; ++l) {
    h->boff.push_back(off);
    off += h->sz[l + 1];
  }
  h->nparam = off;
  long nb = 0;
  h->map.nl = h->nl;
  for (int l = 0; l < h->nl; ++l) {
    h->map.off[l] = h->woff[l];
    h->map.boff[l] = nb;
    h->map.in[l] = h->sz[l];
    nb += (long)pad8(h->sz[l]) * h->sz[l + 1];
  }
  h->map.off[h->nl] = nw;
  h->act.assign(h->nl, OAPB_ACT_TANH);
  h->act[h->nl - 1] = OAPB_ACT_LINEAR;
  const size_t fb = sizeof(float) * (size_t)off;
  if (cudaMalloc(&h->w, fb) != cudaSuccess || cudaMalloc(&h->g, fb) != cudaSuccess ||
      cudaMalloc(&h->m1, fb) != cudaSuccess || cudaMalloc(&h->m2, fb) != cudaSuccess ||
      cudaMalloc(&h->wb, sizeof(__nv_bfloat16) * (size_t)nb) != cudaSuccess ||
      cudaMalloc(&h->loss, sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    delete h;
    return OAPB_ERR_NOMEM;
  }
  cudaMemset(h->m1, 0, fb);
  cudaMemset(h->m2, 0, fb);
  cudaMemset(h->g, 0, fb);
  cudaMemset(h->wb, 0, sizeof(__nv_bfloat16) * (size_t)nb);
  // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases
  for (int l = 0; l < h->nl; ++l) {
    const long len = (long)h->sz[l] * h->sz[l + 1];
    k_init_uniform<<<grid_for(len, 256), 256>>>(h->w + h->woff[l], len, 1.0f / sqrtf((float)h->sz[l]),
                                                 seed * 1315423911ull + l);
  }
  cudaMemset(h->w + nw, 0, sizeof(float) * (size_t)(off - nw));
  k_weights_bf16<<<grid_for(nw, 256), 256>>>(h->w, h->wb, h->map);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    delete h;
    return OAPB_ERR_CUDA;
  }
  *out = h;
  return OAPB_OK;
}

int oapb_mlp_destroy(oapb_mlp* h) {
  if (!h) return OAPB_ERR_ARG;
  cudaDeviceSynchronize();
  free_acts(h);
  cudaFree(h->w);
  cudaFree(h->g);
  cudaFree(h->m1);
  cudaFree(h->m2);
  cudaFree(h->wb);
  cudaFree(h->loss);
  delete h;
  return OAPB_OK;
}

uint64_t oapb_mlp_num_params(const oapb_mlp* h) { return h ? (uint64_t)h->nparam : 0; }

int oapb_mlp_forward(oapb_mlp* h, const float* x, uint32_t batch, float* y, void* stream) {
  if (!h || !x || batch == 0) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int rc = forward_impl(h, x, (int)batch, s);
  if (rc) return rc;
  if (y && cudaMemcpyAsync(y, h->hf[h->nl - 1], sizeof(float) * (size_t)batch * h->sz[h->nl],
                           cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return OAPB_ERR_CUDA;
  return OAPB_OK;
}

// Forward + backward of loss = 1/(2B) sum (y - target)^2; gradients (FP32,
// same packing as the parameters) stay in the handle.  *loss_out (host,
// may be NULL) receives the loss (synchronises the stream).
int oapb_mlp_backward(oapb_mlp* h, const float* x, const float* target, uint32_t batch, double* loss_out,
                      void* stream) {
  if (!h || !x || !target || batch == 0) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int B = (int)batch;
  if (cudaMemsetAsync(h->loss, 0, sizeof(double), s) != cudaSuccess) return OAPB_ERR_CUDA;
  int rc = forward_impl(h, x, B, s);
  if (rc) return rc;
  const int L = h->nl;
  int cur = 0;  // dZ of the layer at hand
  launch_dependent(k_out_grad, dim3(grid_for((long)B * pad8(h->sz[L]), 256, kNumSMs * 8)), dim3(256), 0, s,
                   (const float*)h->hf[L - 1], target, (const float*)h->zf[L - 1], h->act[L - 1], B, h->sz[L],
                   h->dAb[0], pad8(h->sz[L]), h->dA[0], h->loss);
  for (int l = L - 1; l >= 0; --l) {
    const int in = h->sz[l], out = h->sz[l + 1];
    // weight gradient dW[o][i] = sum_b dZ[b][o] X[b][i], bias gradient beside it
    LayerArgs g{};
    g.A = h->dAb[cur];
    g.lda = pad8(out);
    g.B = h->hb[l];
    g.ldb = pad8(in);
    g.M = out;
    g.N = in;
    g.K = B;
    g.C = h->g + h->woff[l];
    g.dZ = h->dA[cur];
    g.db = h->g + h->boff[l];
    if ((rc = layer<0, false, false>(g, s))) return rc;
    if (l == 0) break;
    // data gradient dX[b][i] = sum_o dZ[b][o] W[o][i], through layer l - 1's
    // activation: dZ of that layer
    LayerArgs d{};
    d.A = h->dAb[cur];
    d.lda = pad8(out);
    d.B = h->wb + h->map.boff[l];
    d.ldb = pad8(in);
    d.M = B;
    d.N = in;
    d.K = out;
    d.C = h->dA[cur ^ 1];
    d.Cb = h->dAb[cur ^ 1];
    d.ldcb = pad8(in);
    d.H = h->hf[l - 1];
    d.Zin = h->zf[l - 1];
    d.act = h->act[l - 1];
    if ((rc = layer<2, true, false>(d, s))) return rc;
    cur ^= 1;
  }
  if (cudaGetLastError() != cudaSuccess) return OAPB_ERR_CUDA;
  if (loss_out) {
    if (cudaMemcpyAsync(loss_out, h->loss, sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return OAPB_ERR_CUDA;
  }
  return OAPB_OK;
}

int oapb_mlp_adam_step(oapb_mlp* h, float lr, void* stream) {
  if (!h || !(lr > 0)) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  h->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)h->step), c2 = 1.f - powf(b2, (float)h->step);
  launch_dependent(k_adam, dim3(grid_for(h->nparam, 256)), dim3(256), 0, s, h->w, (const float*)h->g, h->m1, h->m2,
                   h->nparam, lr, b1, b2, 1e-8f, c1, c2, h->wb, h->map);
  return cudaGetLastError() == cudaSuccess ? OAPB_OK : OAPB_ERR_CUDA;
}

// which: 0 parameters (FP32 masters), 1 gradients; dst/src device or host
int oapb_mlp_copy(oapb_mlp* h, int which, float* dst, void* stream) {
  if (!h || !dst || which < 0 || which > 1) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(dst, which ? h->g : h->w, sizeof(float) * (size_t)h->nparam, cudaMemcpyDefault, s) !=
          cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return OAPB_ERR_CUDA;
  return OAPB_OK;
}

int oapb_mlp_set_params(oapb_mlp* h, const float* src, void* stream) {
  if (!h || !src) return OAPB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(h->w, src, sizeof(float) * (size_t)h->nparam, cudaMemcpyDefault, s) != cudaSuccess)
    return OAPB_ERR_CUDA;
  k_weights_bf16<<<grid_for(h->nparam, 256), 256, 0, s>>>(h->w, h->wb, h->map);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return OAPB_ERR_CUDA;
  return OAPB_OK;
}

int oapb_mlp_set_activations(oapb_mlp* h, const int32_t* acts, uint32_t count) {
  if (!h || !acts || count != (uint32_t)h->nl) return OAPB_ERR_ARG;
  for (uint32_t l = 0; l < count; ++l)
    if (acts[l] < OAPB_ACT_LINEAR || acts[l] > OAPB_ACT_SIN) return OAPB_ERR_ARG;
  for (uint32_t l = 0; l < count; ++l) h->act[l] = acts[l];
  return OAPB_OK;
}

int oapb_mlp_get_activations(const oapb_mlp* h, int32_t* acts, uint32_t count) {
  if (!h || !acts || count != (uint32_t)h->nl) return OAPB_ERR_ARG;
  for (uint32_t l = 0; l < count; ++l) acts[l] = h->act[l];
  return OAPB_OK;
}

uint32_t oapb_mlp_num_layers(const oapb_mlp* h, uint32_t* sizes) {
  if (!h) return 0;
  if (sizes)
    for (int i = 0; i <= h->nl; ++i) sizes[i] = (uint32_t)h->sz[i];
  return (uint32_t)h->nl;
}

// File (the reference's matrix format, matio.cuh): sizes (1 column x
// nlayers + 1 rows), then per layer its weights (in columns x out rows) and
// biases (1 column x out rows), FP64 values of the FP32 master weights, and
// last the layers' activations (1 column x nlayers rows, oapb_activation
// values; a file without it loads with the default activations).
int oapb_mlp_save(oapb_mlp* h, const char* path) {
  if (!h || !path) return OAPB_ERR_ARG;
  std::vector<float> p((size_t)h->nparam);
  int rc = oapb_mlp_copy(h, 0, p.data(), nullptr);
  if (rc) return rc;
  std::vector<char> payload;
  HostMat sz;
  sz.columns = 1;
  sz.rows = (uint32_t)(h->nl + 1);
  for (int v : h->sz) sz.re.push_back((double)v);
  matio_append(payload, sz);
  for (int l = 0; l < h->nl; ++l) {
    HostMat W, bv;
    W.columns = (uint32_t)h->sz[l];
    W.rows = (uint32_t)h->sz[l + 1];
    W.re.assign(p.begin() + h->woff[l], p.begin() + h->woff[l] + (long)W.columns * W.rows);
    bv.columns = 1;
    bv.rows = W.rows;
    bv.re.assign(p.begin() + h->boff[l], p.begin() + h->boff[l] + W.rows);
    matio_append(payload, W);
    matio_append(payload, bv);
  }
  HostMat acts;
  acts.columns = 1;
  acts.rows = (uint32_t)h->nl;
  for (int a : h->act) acts.re.push_back((double)a);
  matio_append(payload, acts);
  return matio_write_file(path, payload);
}

int oapb_mlp_load(oapb_mlp** out, const char* path, uint64_t seed) {
  if (!out || !path) return OAPB_ERR_ARG;
  std::vector<char> payload;
  int rc = matio_read_file(path, &payload);
  if (rc) return rc;
  size_t off = 0;
  HostMat sz;
  if (!matio_parse(payload, off, &sz) || sz.columns != 1 || sz.rows < 2 || sz.rows > 9) return OAPB_ERR_ARG;
  std::vector<uint32_t> sizes;
  for (double v : sz.re) {
    if (!(v >= 1 && v < 1e9)) return OAPB_ERR_ARG;
    sizes.push_back((uint32_t)v);
  }
  const int nl = (int)sizes.size() - 1;
  std::vector<HostMat> Ws(nl), bs(nl);
  for (int l = 0; l < nl; ++l) {
    if (!matio_parse(payload, off, &Ws[l]) || !matio_parse(payload, off, &bs[l])) return OAPB_ERR_ARG;
    if (Ws[l].columns != sizes[l] || Ws[l].rows != sizes[l + 1] || bs[l].columns != 1 || bs[l].rows != sizes[l + 1])
      return OAPB_ERR_ARG;
  }
  std::vector<int32_t> acts;
  HostMat am;
  if (off < payload.size()) {
    if (!matio_parse(payload, off, &am) || am.columns != 1 || am.rows != (uint32_t)nl) return OAPB_ERR_ARG;
    for (double v : am.re) {
      if (!(v >= OAPB_ACT_LINEAR && v <= OAPB_ACT_SIN) || v != (double)(int)v) return OAPB_ERR_ARG;
      acts.push_back((int32_t)v);
    }
  }
  oapb_mlp* h = nullptr;
  if ((rc = oapb_mlp_create(&h, sizes.data(), (uint32_t)nl, seed))) return rc;
  if (!acts.empty()) oapb_mlp_set_activations(h, acts.data(), (uint32_t)nl);
  std::vector<float> p((size_t)h->nparam);
  for (int l = 0; l < nl; ++l) {
    for (size_t e = 0; e < Ws[l].re.size(); ++e) p[h->woff[l] + e] = (float)Ws[l].re[e];
    for (size_t e = 0; e < bs[l].re.size(); ++e) p[h->boff[l] + e] = (float)bs[l].re[e];
  }
  if ((rc = oapb_mlp_set_params(h, p.data(), nullptr))) {
    oapb_mlp_destroy(h);
    return rc;
  }
  *out = h;
  return OAPB_OK;
}

}  // extern "C"
