// bf16 GEMM for at most 64 tokens and weights of a few megabytes: D[M, N] = X[M, K] * W[N, K]^T (+bias), and the gated-MLP
// up-projection silu(X Wg^T) * (X Wu^T) of the stacked weight [Wg; Wu].
//
// What bounds these calls is latency, not bandwidth: the projections of a 0.5B model hold 1.6 to 17 MB (0.3 to 2.7 us of HBM time) and a
// decode step makes 96 of them. The tcgen05 kernel for few tokens spends about 10 us on each: TMEM allocation, barrier and descriptor
// set-up, a cooperative launch, and a K split whose partial sums travel through global memory with a grid-wide wait. Here
//   * a warp keeps its weights in registers: a lane loads 32 contiguous bytes of two rows (one 128-byte line per row and quad), all
//     blocks of its first batch before the first is used, and feeds them to mma.sync m16n8k16 as they are. The contraction index is
//     permuted alike in both operands (a lane's 16 consecutive elements are the k slots of four MMAs), so neither needs shared memory;
//   * the eight warps of a CTA split K in blocks of 64; with few row tiles a cluster of 2 to 8 CTAs splits it further and sums through
//     distributed shared memory: no workspace, no counters, no second launch;
//   * the gate and up rows of one output column meet in one CTA, whose epilogue applies the activation (rounded to bf16 in between, as
//     the two launches it replaces did).
// mma.sync cannot reach the tensor peak, but at 8 to 64 tokens the work is 2 to 16 MMAs per 2 KB of weights.
// Measured in a captured graph with weights from HBM, 4 tokens, against the tcgen05 kernel for few tokens (and the activation's launch):
// 1152 x 896 8.4 -> 2.5 us, 9728 x 896 gated 11.0 -> 5.6 us, 896 x 4864 11.8 -> 5.8 us, 5120 x 2048 12.1 -> 6.6 us, 4608 x 3584
// 13.6 -> 9.0 us (floor at the copy rate: 0.3, 2.7, 1.4, 3.3, 5.2 us). Where it stops being the better one: vb_few_tokens_better.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "launchers.h"
#include "tcgen05_common.cuh"

namespace vb {
namespace cg = cooperative_groups;

constexpr int FT_WARPS = 8, FT_THREADS = 32 * FT_WARPS;
constexpr int FT_KB = 64;          // K per block
constexpr int FT_MAX_TOKENS = 64, FT_MAX_GATED = 16;

struct FewTokensParams {
  const __nv_bfloat16* X;
  const __nv_bfloat16* W;
  const __nv_bfloat16* bias;  // [N] or null
  __nv_bfloat16* D;
  long long ldx, ldw, ldd;
  int M, N, K;                // N: output columns (SWIGLU: I; W has 2 I rows)
};

__device__ __forceinline__ uint4 ft_ldw(const __nv_bfloat16* p) {  // weights: read once
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void ft_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: tiles of 8 tokens. MT: tiles of 16 weight rows (SWIGLU: the first is gate rows, the second up rows). U: blocks of 64 whose weights
// a warp has in flight together.
template <int NT, int MT, bool SWIGLU, int U>
__global__ void __launch_bounds__(FT_THREADS, U == 1 ? 3 : 2)
few_tokens_kernel(const FewTokensParams p) {
  static_assert(!SWIGLU || MT == 2, "a gate and an up tile");
  constexpr int ROWS = 16 * MT, TOK = 8 * NT, PITCH = TOK + 1;
  extern __shared__ float s_part[];                   // [FT_WARPS][ROWS][PITCH]; the CTA's sum ends up in the first
  cg::cluster_group cluster = cg::this_cluster();
  const int cl = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int tile = blockIdx.x / cl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const int row0 = tile * (SWIGLU ? 16 : ROWS);
  const int nb = (p.K + FT_KB - 1) / FT_KB;

  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;

  // rows and tokens past the end read the last valid one; what comes of them is not stored
  const __nv_bfloat16* wrow[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = min(row0 + (SWIGLU ? 0 : 16 * m) + 8 * h + g, p.N - 1) + (SWIGLU && m == 1 ? p.N : 0);
      wrow[m][h] = p.W + static_cast<long long>(r) * p.ldw + tig * 16;
    }
  const __nv_bfloat16* xrow[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xrow[n] = p.X + static_cast<long long>(min(8 * n + g, p.M - 1)) * p.ldx + tig * 16;

  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int b0 = rank * FT_WARPS + warp; b0 < nb; b0 += U * cl * FT_WARPS) {
    uint4 w[U][MT][2][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (b0 + u * cl * FT_WARPS) * FT_KB;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 2; ++c) w[u][m][h][c] = k + tig * 16 + c * 8 < p.K ? ft_ldw(wrow[m][h] + k + c * 8) : zero;  // K % 8 == 0
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (b0 + u * cl * FT_WARPS) * FT_KB;
      if (k >= p.K) break;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        uint4 x[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) x[c] = k + tig * 16 + c * 8 < p.K ? *reinterpret_cast<const uint4*>(xrow[n] + k + c * 8) : zero;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint4 &lo = w[u][m][0][c], &hi = w[u][m][1][c];
            ft_mma(acc[m][n], lo.x, hi.x, lo.y, hi.y, x[c].x, x[c].y);
            ft_mma(acc[m][n], lo.z, hi.z, lo.w, hi.w, x[c].z, x[c].w);
          }
      }
    }
  }

  // sum over the warps, then over the cluster; every CTA of the cluster finishes its share of the tile
  float* mine = s_part + warp * (ROWS * PITCH);
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) mine[(16 * m + g + 8 * (i >> 1)) * PITCH + 8 * n + 2 * tig + (i & 1)] = acc[m][n][i];
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS * TOK; i += FT_THREADS) {
    float* at = s_part + (i / TOK) * PITCH + i % TOK;
    float s = at[0];
#pragma unroll
    for (int w = 1; w < FT_WARPS; ++w) s += at[w * (ROWS * PITCH)];
    at[0] = s;
  }
  if (cl > 1) cluster.sync();
  else __syncthreads();
  auto sum = [&](int r, int t) {
    const int o = r * PITCH + t;
    if (cl == 1) return s_part[o];
    float s = 0.f;
    for (int c = 0; c < cl; ++c) s += cluster.map_shared_rank(s_part, c)[o];
    return s;
  };
  constexpr int OUT = SWIGLU ? 16 : ROWS;  // output columns of the tile, two per thread and step
  for (int i = rank * FT_THREADS + threadIdx.x; i < OUT / 2 * TOK; i += cl * FT_THREADS) {
    const int t = i / (OUT / 2), r = (i % (OUT / 2)) * 2, col = row0 + r;
    if (t >= p.M || col >= p.N) continue;  // N is even
    float a = sum(r, t), b = sum(r + 1, t);
    if constexpr (SWIGLU) {
      a = __bfloat162float(__float2bfloat16(a));
      b = __bfloat162float(__float2bfloat16(b));
      const float ua = __bfloat162float(__float2bfloat16(sum(16 + r, t))), ub = __bfloat162float(__float2bfloat16(sum(17 + r, t)));
      a = a / (1.f + __expf(-a)) * ua;
      b = b / (1.f + __expf(-b)) * ub;
    } else if (p.bias != nullptr) {
      a += __bfloat162float(p.bias[col]);
      b += __bfloat162float(p.bias[col + 1]);
    }
    *reinterpret_cast<__nv_bfloat162*>(p.D + static_cast<long long>(t) * p.ldd + col) = __floats2bfloat162_rn(a, b);
  }
  if (cl > 1) cluster.sync();  // a peer may still read this CTA's sums
}

template <int NT, int MT, bool SWIGLU, int U>
static cudaError_t launch_few_tokens(const FewTokensParams& p, int tiles, int cl, cudaStream_t stream) {
  auto kern = few_tokens_kernel<NT, MT, SWIGLU, U>;
  constexpr int smem = FT_WARPS * 16 * MT * (8 * NT + 1) * 4;
  static_assert(smem <= 48 * 1024, "shared memory without an attribute");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles) * cl);
  cfg.blockDim = dim3(FT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace vb

using namespace vb;

// Whether this kernel is the better one for M tokens (measured, weights from HBM; tcgen05 kernel -> this one):
//   gated, 16 tokens: 9728 x 896 11.3 -> 7.6 us; 32 tokens 11.3 -> 11.4 us; 37888 x 3584 at 4 / 8 / 16 tokens 47.7 -> 43.3,
//   48.0 -> 45.6, 48.6 -> 52.7 us;
//   plain, up to 32 tokens: 896 x 4864 12.0 -> 8.1, 5120 x 2048 12.3 -> 10.3, 4608 x 3584 13.8 -> 11.4 us; 3584 x 18944 (136 MB)
//   30.5 -> 41 us, and at 8 tokens 29.8 -> 30.9 us: there the weights of a tile are read through more, smaller requests;
//   64 tokens: 1152 x 896 9.9 -> 5.7, 128 x 2048 8.8 -> 5.8, 896 x 4864 12.4 -> 11.8, 2048 x 4096 12.7 -> 13.5 us: every CTA reads all
//   tokens through its L1, which costs as much as the weights.
extern "C" int vb_few_tokens_better(int M, int N, int K, int swiglu) {
  const long long bytes = 2LL * N * K * (swiglu ? 2 : 1);
  if (swiglu) return M <= 8 || (M <= FT_MAX_GATED && bytes <= (40LL << 20));
  return (M <= 32 && bytes <= (40LL << 20)) || (M <= FT_MAX_TOKENS && bytes <= (4LL << 20));
}

// swiglu: N is the width I of the activation, W has 2 I rows, M at most 16 (the rule above takes it no further). Pointers 16-byte aligned (D: 4), ldx, ldw and K multiples of 8, ldd and N even.
extern "C" int vb_gemm_few_tokens(const void* X, const void* W, void* D, const void* bias, int M, int N, int K, long long ldx, long long ldw,
                                  long long ldd, int swiglu, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || M > (swiglu ? FT_MAX_GATED : FT_MAX_TOKENS)) return -1;
  if ((K % 8) || (N % 2) || (ldx % 8) || (ldw % 8) || (ldd % 2)) return -1;
  if (((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15) || (reinterpret_cast<uintptr_t>(D) & 3)) return -2;
  FewTokensParams p{};
  p.X = reinterpret_cast<const __nv_bfloat16*>(X); p.W = reinterpret_cast<const __nv_bfloat16*>(W);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.D = reinterpret_cast<__nv_bfloat16*>(D);
  p.ldx = ldx; p.ldw = ldw; p.ldd = ldd; p.M = M; p.N = N; p.K = K;
  const int tiles = (N + 15) / 16, nb = (K + FT_KB - 1) / FT_KB;
  // split K over a cluster while every warp keeps a block and there are fewer than one and a half CTAs per SM: 896 x 4864 at 64 tokens 20.0 ->
  // 11.9 us with the split; up to two per SM the second CTA's exchange costs more than its loads hide (4608 x 3584 at 32 tokens 11.8 -> 18.2 us)
  int cl = 1;
  while (cl < 8 && 2 * tiles * cl < 3 * num_sms() && nb >= 2 * cl * FT_WARPS) cl *= 2;
  // two CTAs per SM with two blocks per warp in flight, or three with one where that makes it a single wave (5120 x 2048, 32 tokens:
  // 320 CTAs, 12.4 us with two, 10.3 us with three); the gated product has two tiles per warp and takes three throughout
  const int ctas = tiles * cl, sms = num_sms();
  const bool three = (ctas > 2 * sms && ctas <= 3 * sms);
  cudaError_t e;
  auto plain = [&](auto nt) {
    constexpr int NT = decltype(nt)::value;
    return three ? launch_few_tokens<NT, 1, false, 1>(p, tiles, cl, stream) : launch_few_tokens<NT, 1, false, 2>(p, tiles, cl, stream);
  };
  if (swiglu) e = M <= 8 ? launch_few_tokens<1, 2, true, 1>(p, tiles, cl, stream) : launch_few_tokens<2, 2, true, 1>(p, tiles, cl, stream);
  else if (M <= 8) e = plain(std::integral_constant<int, 1>{});
  else if (M <= 16) e = plain(std::integral_constant<int, 2>{});
  else if (M <= 32) e = plain(std::integral_constant<int, 4>{});
  else e = plain(std::integral_constant<int, 8>{});
  return static_cast<int>(e);
}
