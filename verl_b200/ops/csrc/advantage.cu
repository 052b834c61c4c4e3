// Advantage estimators on the device: GRPO group-normalised outcome advantage and GAE (reverse scan with
// mask carry-through) plus masked whitening.  Semantics follow verl/trainer/ppo/core_algos.py:216-331.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace vb {
int num_sms();

// scores[b] = sum_t rewards[b,t]; one block per row. With `stats` (zeroed by the caller) also stats[g] += {sum, sum of squares, count}, in
// double: sums of fp32 scores and of their squares are then good for a variance far below the square of the mean.
template <typename I>
__global__ void __launch_bounds__(128)
grpo_scores_kernel(const float* __restrict__ rewards, const I* __restrict__ group, int L, float* __restrict__ scores,
                   double* __restrict__ stats) {
  __shared__ float red[4];
  const float* row = rewards + static_cast<long long>(blockIdx.x) * L;
  float s = 0.f;
  for (int t = threadIdx.x; t < L; t += 128) s += row[t];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float tot = red[0] + red[1] + red[2] + red[3];
    scores[blockIdx.x] = tot;
    if (stats) {
      double* st = stats + 3 * static_cast<long long>(group[blockIdx.x]);
      atomicAdd(st, static_cast<double>(tot));
      atomicAdd(st + 1, static_cast<double>(tot) * tot);
      atomicAdd(st + 2, 1.0);
    }
  }
}

// Sums of a and b over the block.
__device__ __forceinline__ void grpo_block_sum(double& a, int& b, double (&ra)[4], int (&rb)[4]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  b = __reduce_add_sync(0xffffffffu, b);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    ra[threadIdx.x >> 5] = a;
    rb[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  a = ra[0] + ra[1] + ra[2] + ra[3];
  b = rb[0] + rb[1] + rb[2] + rb[3];
}

// adv[b,t] = (score - mean_g) / (std_g + eps) * mask[b,t]   (unbiased std; singleton group: mean 0, std 1). Without `stats` a row's
// block finds the members of its group among the B scores itself: the mean first, then the squares around it, with neither a zeroed scratch
// nor atomics. That scan is quadratic in B over the whole grid, so it is taken up to GRPO_SCAN_ROWS. Mean and variance are formed in double
// on both ways: a group's scores can lie as close together as fp32 can tell (50 +- 0.01: with fp32 sums the advantages were off by 2e-4 with
// the scan, and meaningless from the atomics).
template <typename I>
__global__ void __launch_bounds__(128)
grpo_adv_kernel(const float* __restrict__ scores, const I* __restrict__ group, const double* __restrict__ stats,
                const float* __restrict__ mask, int B, int L, float eps, int norm_by_std, float* __restrict__ adv) {
  __shared__ double red[4];
  __shared__ int red_n[4];
  const int b = blockIdx.x;
  const I g = group[b];
  int n = 0;
  double sum = 0.0;
  if (stats) {
    n = static_cast<int>(stats[3 * static_cast<long long>(g) + 2]);
    sum = stats[3 * static_cast<long long>(g)];
  } else {
    for (int i = threadIdx.x; i < B; i += 128)
      if (group[i] == g) {
        n += 1;
        sum += scores[i];
      }
    grpo_block_sum(sum, n, red, red_n);
  }
  double mean = 0.0, sd = 1.0;
  if (n > 1) {
    mean = sum / n;
    double sq = 0.0;
    if (stats) {
      sq = stats[3 * static_cast<long long>(g) + 1] - n * mean * mean;
      if (sq < 0.0) sq = 0.0;  // (NaN stays)
    } else {
      int unused = 0;
      for (int i = threadIdx.x; i < B; i += 128)
        if (group[i] == g) sq += (scores[i] - mean) * (scores[i] - mean);
      grpo_block_sum(sq, unused, red, red_n);
    }
    sd = sqrt(sq / (n - 1));
  }
  const float a = static_cast<float>(norm_by_std ? (scores[b] - mean) / (sd + eps) : scores[b] - mean);
  const long long row = static_cast<long long>(b) * L;
  for (int t = threadIdx.x; t < L; t += 128) adv[row + t] = a * mask[row + t];
}

// One step of GAE, from the later state (value and advantage of the next unmasked token) to the earlier one, is an affine map
//   n' = p n + u,   l' = q n + s l + w
// with p = 1 - mask, u = mask * v, q = mask * gamma, s = mask * gamma * lambda + 1 - mask, w = mask * (r - v). Such maps compose to
// maps of the same form, so the reverse scan over time is a prefix scan.
struct GaeMap {
  float p, u, q, s, w;
};
__device__ __forceinline__ GaeMap gae_after(const GaeMap& e, const GaeMap& l) {  // the map `l` (later tokens) first, then `e`
  return {e.p * l.p, e.p * l.u + e.u, e.q * l.p + e.s * l.q, e.s * l.s, e.q * l.u + e.s * l.w + e.w};
}
__device__ __forceinline__ GaeMap gae_shfl_down(const GaeMap& m, int o) {
  return {__shfl_down_sync(0xffffffffu, m.p, o), __shfl_down_sync(0xffffffffu, m.u, o), __shfl_down_sync(0xffffffffu, m.q, o),
          __shfl_down_sync(0xffffffffu, m.s, o), __shfl_down_sync(0xffffffffu, m.w, o)};
}

constexpr int GAE_PER = 4;           // consecutive tokens per thread
constexpr int GAE_BLOCKS_PER_SM = 8;

// A block takes whole rows and walks a row from its end in tiles of blockDim * 4 tokens: every thread composes the maps of its four
// tokens, a scan over the block gives the state behind them, and the four tokens are then stepped through. 512 x 1024 tokens: 267 us with
// one thread per row (serial loads of the whole row, uncoalesced) -> 8 us for the scan and the whitening (13.8 us the whole call, 284 before); the bytes alone are 1.6 us, what is left is one
// row's chain of load, scan and store. `part` (null: no whitening) gets the block's masked sums of the advantages: sum, sum of
// squares, count.
__global__ void __launch_bounds__(256)
gae_kernel(const float* __restrict__ rewards, const float* __restrict__ values, const float* __restrict__ mask, int B, int L, float gamma,
           float lam, float* __restrict__ adv, float* __restrict__ ret, double* __restrict__ part) {
  __shared__ GaeMap warp_map[8];
  __shared__ float carry[2];
  __shared__ double red[8][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int tile = blockDim.x * GAE_PER;
  float s1 = 0.f, s2 = 0.f, s0 = 0.f;
  for (int b = blockIdx.x; b < B; b += gridDim.x) {
    const long long row = static_cast<long long>(b) * L;
    float n_in = 0.f, l_in = 0.f;  // the state behind the tile
    for (int t1 = ((L + tile - 1) / tile) * tile; t1 > 0; t1 -= tile) {
      const int t0 = t1 - tile + threadIdx.x * GAE_PER;
      float r[GAE_PER], v[GAE_PER], m[GAE_PER];
#pragma unroll
      for (int j = 0; j < GAE_PER; ++j) {
        const bool in = t0 + j < L;
        r[j] = in ? rewards[row + t0 + j] : 0.f;
        v[j] = in ? values[row + t0 + j] : 0.f;
        m[j] = in ? mask[row + t0 + j] : 0.f;  // a masked token hands the state through
      }
      GaeMap acc{1.f, 0.f, 0.f, 1.f, 0.f};
#pragma unroll
      for (int j = GAE_PER - 1; j >= 0; --j)
        acc = gae_after({1.f - m[j], m[j] * v[j], m[j] * gamma, m[j] * gamma * lam + 1.f - m[j], m[j] * (r[j] - v[j])}, acc);
      // inclusive scan from the warp's last lane backwards, then over the warps
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const GaeMap later = gae_shfl_down(acc, o);
        if (lane + o < 32) acc = gae_after(acc, later);
      }
      if (lane == 0) warp_map[warp] = acc;
      GaeMap behind = gae_shfl_down(acc, 1);  // of the lanes behind this one
      if (lane == 31) behind = {1.f, 0.f, 0.f, 1.f, 0.f};
      __syncthreads();
      for (int k = warp + 1; k < warps; ++k) behind = gae_after(behind, warp_map[k]);
      float nextv = behind.p * n_in + behind.u, last = behind.q * n_in + behind.s * l_in + behind.w;
#pragma unroll
      for (int j = GAE_PER - 1; j >= 0; --j) {
        const float cand = r[j] + gamma * nextv - v[j] + gamma * lam * last;
        nextv = v[j] * m[j] + (1.f - m[j]) * nextv;
        last = cand * m[j] + (1.f - m[j]) * last;
        if (t0 + j < L) {
          adv[row + t0 + j] = last;
          ret[row + t0 + j] = last + v[j];
          s1 += last * m[j];
          s2 += last * last * m[j];
          s0 += m[j];
        }
      }
      if (threadIdx.x == 0) {
        carry[0] = nextv;
        carry[1] = last;
      }
      __syncthreads();
      n_in = carry[0];
      l_in = carry[1];
    }
  }
  if (!part) return;
  double d[3] = {s1, s2, s0};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d[k] += __shfl_xor_sync(0xffffffffu, d[k], o);
    if (lane == 0) red[warp][k] = d[k];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int k = 0; k < warps; ++k) t += red[k][threadIdx.x];
    part[blockIdx.x * 3 + threadIdx.x] = t;
  }
}

// x <- (x - mean) * rsqrt(var + 1e-8), unbiased variance over the unmasked tokens. Every block folds the partial sums of the scan
// (at most eight per SM) itself, in one order: no memset, no atomics, the same bits every time.
__global__ void __launch_bounds__(256)
whiten_kernel(float* __restrict__ x, long long n, const double* __restrict__ part, int nparts) {
  __shared__ double red[8][3];
  __shared__ float mw[2];
  double d[3] = {0, 0, 0};
  for (int i = threadIdx.x; i < nparts; i += blockDim.x)
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] += part[i * 3 + k];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d[k] += __shfl_xor_sync(0xffffffffu, d[k], o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = d[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[3] = {0, 0, 0};
    for (int k = 0; k < 8; ++k)
      for (int j = 0; j < 3; ++j) t[j] += red[k][j];
    const double c = t[2], mean = t[0] / (c + 1e-8);
    const double var = fmax(t[1] / (c + 1e-8) - mean * mean, 0.0) * (c / fmax(c - 1.0, 1.0));
    mw[0] = static_cast<float>(mean);
    mw[1] = static_cast<float>(1.0 / sqrt(var + 1e-8));
  }
  __syncthreads();
  const float mean = mw[0], scale = mw[1];
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) x[i] = (x[i] - mean) * scale;
}

}  // namespace vb

using namespace vb;

extern "C" {

// Up to this many rows the scan of grpo_adv_kernel is the cheaper way (320 x 2048: 21.5 us for the call with memset, conversion of the
// ids and atomics, 12.6 us with the scan; at 2560 rows the scan's 157 MB of L2 reads take longer than the atomics).
constexpr int GRPO_SCAN_ROWS = 1024;
int vb_grpo_needs_stats(int B) { return B > GRPO_SCAN_ROWS; }

// group: int32 or int64 ids (group64); ids in [0, num_groups). stats: 3 * num_groups doubles (zeroed here) when vb_grpo_needs_stats.
int vb_grpo_advantage(const float* rewards, const float* mask, const void* group, int group64, int B, int L, int num_groups, float eps,
                      int norm_by_std, float* scores, double* stats, float* adv, cudaStream_t s) {
  if (B == 0) return 0;
  if (vb_grpo_needs_stats(B))
    cudaMemsetAsync(stats, 0, sizeof(double) * 3 * num_groups, s);
  else
    stats = nullptr;
  if (group64) {
    const long long* g = static_cast<const long long*>(group);
    grpo_scores_kernel<<<B, 128, 0, s>>>(rewards, g, L, scores, stats);
    grpo_adv_kernel<<<B, 128, 0, s>>>(scores, g, stats, mask, B, L, eps, norm_by_std, adv);
  } else {
    const int* g = static_cast<const int*>(group);
    grpo_scores_kernel<<<B, 128, 0, s>>>(rewards, g, L, scores, stats);
    grpo_adv_kernel<<<B, 128, 0, s>>>(scores, g, stats, mask, B, L, eps, norm_by_std, adv);
  }
  return static_cast<int>(cudaGetLastError());
}

// Blocks of the scan = rows of `part` (3 doubles each). A row's tiles follow one another, so rows are what fills the machine; a block
// is as wide as the row needs, up to 256 threads (1024 tokens per tile).
int vb_gae_blocks(int B) { return B < GAE_BLOCKS_PER_SM * num_sms() ? B : GAE_BLOCKS_PER_SM * num_sms(); }

// Whitening of the advantages over the whole batch (statistics over unmasked tokens, result not re-masked) is applied when `part` is
// given.
int vb_gae(const float* rewards, const float* values, const float* mask, int B, int L, float gamma, float lam, float* adv, float* ret,
           double* part, cudaStream_t s) {
  if (B == 0 || L == 0) return 0;
  const int want = (L + GAE_PER - 1) / GAE_PER;
  const int threads = want >= 256 ? 256 : (want + 31) / 32 * 32;
  gae_kernel<<<vb_gae_blocks(B), threads, 0, s>>>(rewards, values, mask, B, L, gamma, lam, adv, ret, part);
  if (part) {
    const long long n = static_cast<long long>(B) * L;
    // a block per 1024 tokens, four per SM at most: every block folds the partial sums
    const long long want_blocks = (n + 1023) / 1024, most = 4LL * num_sms();
    whiten_kernel<<<static_cast<int>(want_blocks < most ? want_blocks : most), 256, 0, s>>>(adv, n, part, vb_gae_blocks(B));
  }
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
