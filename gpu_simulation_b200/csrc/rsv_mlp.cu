// Warm-start network kernels: a fully connected GELU network in FP32 with
// FP32 accumulation (forward, backward, squared-error loss) and fused Adam
// steps (FP32 for the network, FP64 for circuit angles).
//
// The reference has no learned component; its VQE loop is plain gradient
// descent on the angles (ring_ising/optimizers.py, run by
// ring_ising/runner.py).  The network maps circuit descriptors (h, n, L) to
// initial angles; every energy reported still comes from the simulator.
//
// All matrices are row-major.  A linear layer with K inputs and N outputs
// stores W as N x K followed by b (N).  Shapes are small (batch <= a few
// thousand, widths <= a few hundred), so a product is bound by the latency of
// its depth loop and by how many SMs it reaches.  One CUDA-core GEMM with
// generic strides serves the forward product and both backward products: 32 x 32
// output tiles (a 512 x 256 product is 128 CTAs), the depth split over four
// groups of 64 threads that meet once at the end, the next stage's loads in
// flight during a stage, and what follows a product in its epilogue (bias and
// GELU; GELU's derivative; the bias gradient, which is the row sums of the
// weight gradient's first operand).  A layer's weight gradient and the gradient
// of its input are independent and share a launch.  Where a launch has CTAs to
// spare a cluster of 2 to 8 shares a tile's depth (a weight gradient's is the
// number of rows) and adds its parts through distributed shared memory in its order.  A
// shallow product over many rows gives every thread group a tile of its own instead.  One loss
// and gradient of the 3-256-256-192 network on 512 rows takes 7 launches instead
// of 15, and 71 us against 371 (64 x 64 tiles without prefetch on 16 to 32 CTAs, and column
// sums that one thread added over all rows); its error against 64 bits went
// from 3.4e-7 to 1.0e-7.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "rsv_mlp.h"

namespace rsv {
namespace {

namespace cg = cooperative_groups;

constexpr int kTile = 32;          // output tile (rows x cols)
constexpr int kTileK = 16;         // depth of one shared-memory stage
constexpr int kGroups = 4;         // thread groups sharing the depth
constexpr int kGroupThreads = 64;  // 8 x 8 threads, 4 x 4 outputs each
constexpr int kGemmThreads = kGroups * kGroupThreads;
// CTAs of a launch that shares depths: three a SM.  Loss and gradient on 512 rows,
// us by this limit: none shared 79, 160 75.7, 296 76.9, 400 to 444 70.7, 592 78.6, 900 85.4; on
// 32 rows 50 without and 41 with, on 1024 rows 125 and 109.
constexpr int kMostBlocks = 444;
// A product of small depth and many tiles has nothing to gain from a split depth, and
// pays for its idle groups and their meeting: from kWholeTiles tiles on, one that is
// less than 128 deep gives every group a tile of its own.  Us, split and whole
// (64 x 64 tiles took): 3 -> 64 on 16384 rows (1024 tiles) 14.6 and 11.3 (16), on
// 131072 82 and 17 (18); 3 -> 256 on 131072 320 and 58 (60); 32 -> 256 336 and 123
// (202); 64 -> 256 407 and 224 (386); 96 -> 64 158 and 87 (146); with 512 tiles
// and less the two are equal within 5 %, and the split sum is the more exact one.
// 128 deep and more the split form is the faster one against the 64 x 64 tiles too
// (128 -> 256 636, 754) and stays.  kWholeCtas: resident CTAs that the registers are
// limited for (3 -> 256 on 131072 rows: 2 74, 3 61, 4 58, 5 70).
constexpr int kWholeDepth = 127, kWholeTiles = 1024, kWholeCtas = 4;
constexpr int kPad = kTile + 4;    // 16-byte rows, two-way conflicts at most on the stores

__device__ __forceinline__ float gelu(float z) {
  return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}

// d gelu / dz = Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

struct GemmPair {
  MlpGemm g[2];
  int tiles_n[2], tiles[2];  // column tiles, and all of them
  int log_splits[2], blocks[2];  // log2 of the CTAs (a cluster) that share a tile's depth; all, in whole clusters
};

// How the four groups of a CTA work: on one tile, each with a part of its depth
// (the CTA's, or its cluster's share of it); or each on a tile of its own.
enum class Depth { kSplit, kShared, kWhole };

template <Depth form>
__global__ void __launch_bounds__(kGemmThreads, form == Depth::kWhole ? kWholeCtas : 0) gemm_kernel(const __grid_constant__ GemmPair P) {
  constexpr bool shared_depth = form == Depth::kShared, whole = form == Depth::kWhole;
  __shared__ float stage[kGroups][2][2][kTileK][kPad];  // [group][buffer][A, B][k][m or n]
  __shared__ float rows[kGroups][kTile];
  const int which = static_cast<int>(blockIdx.x) < P.blocks[0] ? 0 : 1;
  const MlpGemm &g = P.g[which];
  const int log_splits = shared_depth ? P.log_splits[which] : 0, splits = 1 << log_splits;
  const int block = static_cast<int>(blockIdx.x) - (which ? P.blocks[0] : 0);
  const int tid = threadIdx.x, group = tid / kGroupThreads, t = tid % kGroupThreads;
  const int tile = whole ? block * kGroups + group : block >> log_splits, share = block & (splits - 1);
  if (tile >= P.tiles[which]) return;  // fills up the last cluster, or the last CTA's groups
  const int m0 = tile / P.tiles_n[which] * kTile, n0 = tile % P.tiles_n[which] * kTile;
  const int tx = t % 8, ty = t / 8;
  const int M = g.M, N = g.N, K = g.K;
  // this group's depth range, whole stages
  const int parts = kGroups * splits;
  const int span = ((K + parts * kTileK - 1) >> (log_splits + 6)) * kTileK;  // 64 = kGroups * kTileK
  const int first = whole ? 0 : (share * kGroups + group) * span, end = whole || first + span >= K ? K : first + span;
  // threads run along the contiguous index of each operand
  const bool ak = g.sak == 1, bk = g.sbk == 1;
  const int a_m = ak ? t / 16 : t % 32, a_k = ak ? t % 16 : t / 32, a_dm = ak ? 4 : 0, a_dk = ak ? 0 : 2;
  const int b_n = bk ? t / 16 : t % 32, b_k = bk ? t % 16 : t / 32, b_dn = bk ? 4 : 0, b_dk = bk ? 0 : 2;
  float ra[8], rb[8];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + a_m + i * a_dm, ka = k0 + a_k + i * a_dk;
      ra[i] = m < M && ka < end ? g.A[m * g.sam + ka * g.sak] : 0.0f;
      const int n = n0 + b_n + i * b_dn, kb = k0 + b_k + i * b_dk;
      rb[i] = n < N && kb < end ? g.B[kb * g.sbk + n * g.sbn] : 0.0f;
    }
  };
  float acc[4][4] = {};
  float row = 0.0f;
  const bool sums = g.row_sums != nullptr && n0 == 0 && t < kTile;
  if (first < end) load(first);
  for (int k0 = first, b = 0; k0 < end; k0 += kTileK, b ^= 1) {
    float(&As)[kTileK][kPad] = stage[group][b][0];
    float(&Bs)[kTileK][kPad] = stage[group][b][1];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      As[a_k + i * a_dk][a_m + i * a_dm] = ra[i];
      Bs[b_k + i * b_dk][b_n + i * b_dn] = rb[i];
    }
    // (two buffers: a thread past this barrier knows that the other's readers,
    // one stage back, are done before it writes that one again)
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kGroupThreads) : "memory");
    if (k0 + kTileK < end) load(k0 + kTileK);
#pragma unroll
    for (int kk = 0; kk < kTileK; ++kk) {
      if (whole && kk % 4 == 0 && k0 + kk >= K) break;  // (a depth of 3 is common)
      const float4 a = *reinterpret_cast<const float4 *>(&As[kk][4 * ty]);
      const float4 c = *reinterpret_cast<const float4 *>(&Bs[kk][4 * tx]);
      const float av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], cv[j], acc[i][j]);
    }
    if (sums)
#pragma unroll
      for (int kk = 0; kk < kTileK; ++kk) row += As[kk][t];
  }
  auto finish = [&](int i, int j, float z) {
    const int m = m0 + i, n = n0 + j;
    if (m >= M || n >= N) return;
    const long long at = static_cast<long long>(m) * N + n;
    if (g.bias != nullptr) z += g.bias[n];
    if (g.Z != nullptr) g.Z[at] = z;
    if (g.gelu) z = gelu(z);
    if (g.gelu_of != nullptr) z *= gelu_grad(g.gelu_of[at]);
    g.C[at] = z;
  };
  if constexpr (whole) {  // straight from the registers: a warp's 16-byte stores are whole lines
    const int n = n0 + 4 * tx;
    const bool vec = N % 4 == 0 && ((reinterpret_cast<size_t>(g.C) | reinterpret_cast<size_t>(g.Z)) & 15) == 0;
    float b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = g.bias != nullptr && n + j < N ? g.bias[n + j] : -0.0f;  // (x + -0 is x)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + 4 * ty + i;
      if (m >= M || n >= N) return;
      const long long at = static_cast<long long>(m) * N + n;
      float z[4], c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        z[j] = acc[i][j] + b[j];
        c[j] = g.gelu ? gelu(z[j]) : z[j];
      }
      if (vec) {
        if (g.Z != nullptr) *reinterpret_cast<float4 *>(g.Z + at) = make_float4(z[0], z[1], z[2], z[3]);
        *reinterpret_cast<float4 *>(g.C + at) = make_float4(c[0], c[1], c[2], c[3]);
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (n + j >= N) break;
        if (g.Z != nullptr) g.Z[at + j] = z[j];
        g.C[at + j] = c[j];
      }
    }
    return;
  }
  // the groups' parts, added in group order
  __syncthreads();
  float *part = &stage[0][0][0][0][0];  // [group][kTile][kTile + 1]
  constexpr int kRow = kTile + 1, kPart = kTile * kRow;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) part[group * kPart + (4 * ty + i) * kRow + 4 * tx + j] = acc[i][j];
  if (sums) rows[group][t] = row;
  __syncthreads();
#pragma unroll
  for (int e = tid; e < kTile * kTile; e += kGemmThreads) {
    const int i = e / kTile, j = e % kTile;
    float *p = part + i * kRow + j;
    const float z = (p[0] + p[kPart]) + (p[2 * kPart] + p[3 * kPart]);
    if (!shared_depth || splits == 1) finish(i, j, z);
    else p[0] = z;  // (only this thread reads the element)
  }
  const bool row_sums = g.row_sums != nullptr && n0 == 0 && tid < kTile;
  if (row_sums) {
    const float z = (rows[0][tid] + rows[1][tid]) + (rows[2][tid] + rows[3][tid]);
    if (shared_depth && splits > 1) rows[0][tid] = z;
    else if (m0 + tid < M) g.row_sums[m0 + tid] = z;
  }
  if (!shared_depth || splits == 1) return;
  // the cluster's shares, added in its order; each CTA finishes some of the rows
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int mine = kTile / splits;
  for (int e = tid; e < mine * kTile; e += kGemmThreads) {
    const int i = share * mine + e / kTile, j = e % kTile;
    float z = 0.0f;
    for (int k = 0; k < splits; ++k) z += *cluster.map_shared_rank(part + i * kRow + j, k);
    finish(i, j, z);
  }
  if (row_sums && share == 0 && m0 + tid < M) {
    float z = 0.0f;
    for (int k = 0; k < splits; ++k) z += *cluster.map_shared_rank(&rows[0][tid], k);
    g.row_sums[m0 + tid] = z;
  }
  cluster.sync();  // the shares stay until they are read
}

// Squared error: dOut = 2 (out - target) / count and the mean, by clusters
// whose CTAs' sums meet in shared memory in CTA order.  One cluster writes the
// mean; of larger arrays every kLossElements (up to kMostLossClusters, which fill
// the SMs) have a cluster, these leave their sums in `partials`, and
// loss_finish_kernel adds them in order: a second launch, so from kOneLossCluster
// elements on.  Us on one cluster and on several: 262144 8.3 and 10.9, 300000 9.3 and
// 10.3, 400000 10.4 and 10.3, 800000 16.7 and 10.3, 3.2 M 49 and 11.6, 12.8 M 436 and 35,
// 51.2 M 1736 and 107 (5.7 TB/s).  With 2^17 elements a cluster 800000 take 10.7 us, with
// 2^18 12.4.
constexpr int kLossThreads = 512, kLossCtas = 8, kMostLossClusters = 36;
constexpr long long kOneLossCluster = 3 << 17, kLossElements = 1 << 16;
__global__ void __launch_bounds__(kLossThreads) mse_kernel(long long count, const float *__restrict__ out,
                                                          const float *__restrict__ target,
                                                          float *__restrict__ dout, float *__restrict__ loss,
                                                          float *__restrict__ partials) {
  __shared__ float red[kLossThreads / 32];
  __shared__ float cta;
  cg::cluster_group cluster = cg::this_cluster();
  float s = 0.0f;
  const float scale = 2.0f / static_cast<float>(count);
  const long long stride = static_cast<long long>(gridDim.x) * kLossThreads;
  const long long start = blockIdx.x * static_cast<long long>(kLossThreads) + threadIdx.x;
  // four at a time where the arrays allow it
  const bool vec = ((reinterpret_cast<size_t>(out) | reinterpret_cast<size_t>(target) | reinterpret_cast<size_t>(dout)) & 15) == 0;
  const long long quads = vec ? count / 4 : 0;
#pragma unroll 4
  for (long long i = start; i < quads; i += stride) {
    const float4 o = reinterpret_cast<const float4 *>(out)[i], t = reinterpret_cast<const float4 *>(target)[i];
    const float4 d = make_float4(o.x - t.x, o.y - t.y, o.z - t.z, o.w - t.w);
    reinterpret_cast<float4 *>(dout)[i] = make_float4(scale * d.x, scale * d.y, scale * d.z, scale * d.w);
    s += fmaf(d.x, d.x, d.y * d.y) + fmaf(d.z, d.z, d.w * d.w);
  }
  for (long long i = 4 * quads + start; i < count; i += stride) {
    const float d = out[i] - target[i];
    dout[i] = scale * d;
    s = fmaf(d, d, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < kLossThreads / 32 ? red[threadIdx.x] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) cta = v;
  }
  cluster.sync();
  if (blockIdx.x % kLossCtas == 0 && threadIdx.x == 0) {
    float total = 0.0f;
    for (int k = 0; k < kLossCtas; ++k) total += *cluster.map_shared_rank(&cta, k);
    if (gridDim.x == kLossCtas) *loss = total / static_cast<float>(count);
    else partials[blockIdx.x / kLossCtas] = total;
  }
  cluster.sync();  // the sums stay until they are read
}

__global__ void loss_finish_kernel(int clusters, long long count, const float *__restrict__ partials,
                                   float *__restrict__ loss) {
  float s = 0.0f;
  for (int k = threadIdx.x; k < clusters; k += 32) s += partials[k];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) *loss = s / static_cast<float>(count);
}

// Adam (Kingma & Ba 2015, bias-corrected), one element per thread.
template <typename T>
__global__ void adam_kernel(long long count, T *__restrict__ p, const T *__restrict__ g,
                            T *__restrict__ m, T *__restrict__ v, T lr, T beta1, T beta2, T eps,
                            T corr1, T corr2) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const T gi = g[i];
    const T mi = beta1 * m[i] + (T(1) - beta1) * gi;
    const T vi = beta2 * v[i] + (T(1) - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / corr1) / (sqrt(vi / corr2) + eps);
  }
}

// One plain gradient-descent step of the VQE loop, device resident (the
// reference's apply_gradient_step, ring_ising/workflows/common.py:23-25, and
// the per-step metrics of run_gradient_descent_loop,
// ring_ising/training/loop.py:93-115): p -= stepsize * g; the step's energy
// and |g| are appended to the histories at *counter, which is then
// incremented (so one captured step can be replayed).  One CTA: the norm is
// reduced in a fixed order.
constexpr int kGdThreads = 256;
__global__ void __launch_bounds__(kGdThreads) gd_step_kernel(long long count, double *__restrict__ p,
                                                            const double *__restrict__ g, double stepsize,
                                                            const double *__restrict__ energy,
                                                            double *__restrict__ energy_hist,
                                                            double *__restrict__ gnorm_hist, int *counter) {
  __shared__ double red[kGdThreads];
  double s = 0.0;
  for (long long i = threadIdx.x; i < count; i += kGdThreads) {
    const double gi = g[i];
    s = fma(gi, gi, s);
    p[i] = __dsub_rn(p[i], __dmul_rn(stepsize, gi));  // params - stepsize * grad, no contraction
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = kGdThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int k = *counter;
    if (energy_hist) energy_hist[k] = *energy;
    if (gnorm_hist) gnorm_hist[k] = sqrt(red[0]);
    *counter = k + 1;
  }
}

int elementwise_grid(long long count) {
  const long long b = (count + 255) / 256;
  return static_cast<int>(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

}  // namespace

cudaError_t mlp_gemm(const MlpGemm *g, int count, cudaStream_t s) {
  GemmPair P{};
  for (int k = 0; k < count && k < 2; ++k) {
    P.g[k] = g[k];
    P.tiles_n[k] = (g[k].N + kTile - 1) / kTile;
    P.tiles[k] = P.tiles_n[k] * ((g[k].M + kTile - 1) / kTile);
  }
  if (count == 1 && g[0].row_sums == nullptr && g[0].gelu_of == nullptr && g[0].K <= kWholeDepth &&
      P.tiles[0] >= kWholeTiles) {
    P.blocks[0] = (P.tiles[0] + kGroups - 1) / kGroups;
    gemm_kernel<Depth::kWhole><<<P.blocks[0], kGemmThreads, 0, s>>>(P);
    return cudaGetLastError();
  }
  // as many CTAs a tile as give every group a stage and keep the launch within kMostBlocks
  int size = 1;
  auto plan = [&](int most) {
    int all = 0;
    for (int k = 0; k < 2; ++k) {
      const int splits = P.g[k].K >= most * kGroups * kTileK ? most : 1;
      P.log_splits[k] = splits == 1 ? 0 : splits == 2 ? 1 : splits == 4 ? 2 : 3;
      P.blocks[k] = (P.tiles[k] * splits + most - 1) / most * most;
      all += P.blocks[k];
    }
    return all;
  };
  for (int most = 2; most <= 8; most *= 2)
    if (plan(most) <= kMostBlocks && (P.log_splits[0] > 0 || P.log_splits[1] > 0)) size = most;
  const int blocks = plan(size);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = static_cast<unsigned>(size);
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = size > 1 ? 1 : 0;
  return size > 1 ? cudaLaunchKernelEx(&cfg, gemm_kernel<Depth::kShared>, P)
                  : cudaLaunchKernelEx(&cfg, gemm_kernel<Depth::kSplit>, P);
}

cudaError_t mlp_mse(long long count, const float *out, const float *target, float *dout, float *partials,
                    float *loss, cudaStream_t s) {
  const long long full = count < kOneLossCluster ? 1 : count / kLossElements;
  const int clusters = full < kMostLossClusters ? static_cast<int>(full) : kMostLossClusters;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * kLossCtas));
  cfg.blockDim = dim3(kLossThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kLossCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, mse_kernel, count, out, target, dout, loss, partials);
  if (e != cudaSuccess || clusters == 1) return e;
  loss_finish_kernel<<<1, 32, 0, s>>>(clusters, count, partials, loss);
  return cudaGetLastError();
}

template <typename T>
cudaError_t adam_step(long long count, T *p, const T *g, T *m, T *v, T lr, T beta1, T beta2, T eps,
                      int step, cudaStream_t s) {
  const T corr1 = T(1) - pow(beta1, static_cast<T>(step));
  const T corr2 = T(1) - pow(beta2, static_cast<T>(step));
  adam_kernel<T><<<elementwise_grid(count), 256, 0, s>>>(count, p, g, m, v, lr, beta1, beta2, eps,
                                                         corr1, corr2);
  return cudaGetLastError();
}

// One Adam step of a device-resident VQE loop with torch.optim.Adam's update
// (bias-corrected, no weight decay): m <- m + (1 - beta1)(g - m),
// v <- beta2 v + (1 - beta2) g^2, p <- p - (lr / c1) m / (sqrt(v) / sqrt(c2) + eps)
// with c_i = 1 - beta_i^t.  The step t is *counter + 1 (read on the device, so
// one captured step can be replayed); the step's energy goes to
// energy_hist[*counter] and *counter is incremented.  One CTA.
__global__ void __launch_bounds__(kGdThreads) adam_vqe_step_kernel(long long count, double *__restrict__ p,
                                                                  const double *__restrict__ g,
                                                                  double *__restrict__ m, double *__restrict__ v,
                                                                  double lr, double beta1, double beta2,
                                                                  double eps, const double *__restrict__ energy,
                                                                  double *__restrict__ energy_hist, int *counter) {
  const int k = *counter;
  const double t = static_cast<double>(k + 1);
  const double c1 = 1.0 - pow(beta1, t), c2s = sqrt(1.0 - pow(beta2, t));
  const double step = lr / c1;
  for (long long i = threadIdx.x; i < count; i += kGdThreads) {
    const double gi = g[i];
    const double mi = m[i] + (1.0 - beta1) * (gi - m[i]);
    const double vi = v[i] * beta2 + (1.0 - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= step * (mi / (sqrt(vi) / c2s + eps));
  }
  __syncthreads();  // every thread has read *counter
  if (threadIdx.x == 0) {
    if (energy_hist) energy_hist[k] = *energy;
    *counter = k + 1;
  }
}

cudaError_t adam_vqe_step(long long count, double *p, const double *g, double *m, double *v, double lr,
                          double beta1, double beta2, double eps, const double *energy, double *energy_hist,
                          int *counter, cudaStream_t s) {
  adam_vqe_step_kernel<<<1, kGdThreads, 0, s>>>(count, p, g, m, v, lr, beta1, beta2, eps, energy, energy_hist,
                                                counter);
  return cudaGetLastError();
}

cudaError_t gd_step(long long count, double *p, const double *g, double stepsize, const double *energy,
                    double *energy_hist, double *gnorm_hist, int *counter, cudaStream_t s) {
  gd_step_kernel<<<1, kGdThreads, 0, s>>>(count, p, g, stepsize, energy, energy_hist, gnorm_hist, counter);
  return cudaGetLastError();
}

template cudaError_t adam_step<float>(long long, float *, const float *, float *, float *, float,
                                      float, float, float, int, cudaStream_t);
template cudaError_t adam_step<double>(long long, double *, const double *, double *, double *,
                                       double, double, double, double, int, cudaStream_t);

}  // namespace rsv
