// Rollout-engine kernels: paged KV-cache append, paged decode attention (GQA-aware, one pass over the
// cache per KV head), and the token sampler (temperature + Gumbel-max with the sampled token's log-prob).
// All are bandwidth-bound: the design goal is one coalesced read of every cache byte per decode step.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace vb {
int num_sms();

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------------------------------------------------ KV append
// k/v: [T, nkv, hd] with row stride ld (elements); slot[t] = physical cache row (block * block_size + off),
// negative slots are skipped.  Cache layout: [num_slots, nkv, hd].
__global__ void kv_append_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                                 long long ldk, long long ldv, const long long* __restrict__ slot,
                                 __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc, int row_elems) {
  const long long t = blockIdx.x;
  const long long s = slot[t];
  if (s < 0) return;
  const uint4* ks = reinterpret_cast<const uint4*>(k + t * ldk);
  const uint4* vs = reinterpret_cast<const uint4*>(v + t * ldv);
  uint4* kd = reinterpret_cast<uint4*>(kc + s * row_elems);
  uint4* vd = reinterpret_cast<uint4*>(vc + s * row_elems);
  for (int i = threadIdx.x; i < (row_elems >> 3); i += blockDim.x) {
    kd[i] = ks[i];
    vd[i] = vs[i];
  }
}

// Decode step, one launch per layer instead of three: rotary embedding of q (in place), rotary embedding of k, and the
// append of the rotated k and of v to the paged cache. qkv is the projection output [T, (nh + 2 nkv) * hd] (row stride ld):
// q heads first, then k heads, then v heads. One block per token; threads cover the rotary pairs of all q and k heads and
// the 16-byte pieces of v. A token whose slot is negative (an inactive sequence) only gets its q rotated.
__global__ void rope_kv_append_kernel(__nv_bfloat16* __restrict__ qkv, long long ld, const int* __restrict__ pos,
                                      const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                      const long long* __restrict__ slot, __nv_bfloat16* __restrict__ kc,
                                      __nv_bfloat16* __restrict__ vc, int nh, int nkv, int hd) {
  const long long t = blockIdx.x;
  const int half = hd >> 1, pairs = half >> 1;  // two rotary pairs per thread
  const int p = pos[t];
  const long long s = slot[t];
  __nv_bfloat16* row = qkv + t * ld;
  const int rot_heads = nh + nkv;
  for (int idx = threadIdx.x; idx < rot_heads * pairs; idx += blockDim.x) {
    const int h = idx / pairs, i = (idx - h * pairs) * 2;
    __nv_bfloat16* base = row + static_cast<long long>(h) * hd;
    const float2 c = *reinterpret_cast<const float2*>(cos_t + static_cast<long long>(p) * half + i);
    const float2 sn = *reinterpret_cast<const float2*>(sin_t + static_cast<long long>(p) * half + i);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(base + i));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(base + half + i));
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x * c.x - b.x * sn.x, a.y * c.y - b.y * sn.y);
    const __nv_bfloat162 hi = __floats2bfloat162_rn(b.x * c.x + a.x * sn.x, b.y * c.y + a.y * sn.y);
    *reinterpret_cast<__nv_bfloat162*>(base + i) = lo;
    *reinterpret_cast<__nv_bfloat162*>(base + half + i) = hi;
    if (h >= nh && s >= 0) {  // a key head: the rotated values also go to the cache
      __nv_bfloat16* kd = kc + s * static_cast<long long>(nkv) * hd + static_cast<long long>(h - nh) * hd;
      *reinterpret_cast<__nv_bfloat162*>(kd + i) = lo;
      *reinterpret_cast<__nv_bfloat162*>(kd + half + i) = hi;
    }
  }
  if (s >= 0) {
    const uint4* vs = reinterpret_cast<const uint4*>(row + static_cast<long long>(nh + nkv) * hd);
    uint4* vd = reinterpret_cast<uint4*>(vc + s * static_cast<long long>(nkv) * hd);
    for (int i = threadIdx.x; i < (nkv * hd) >> 3; i += blockDim.x) vd[i] = vs[i];
  }
}

// RMSNorm of every q and k head, rotary embedding, and optionally the append of k and v to the paged cache, in place in the projection
// output: one warp per (token, head), 16 bytes per lane. Every value is the one that the separate kernels gave, to the bit: the sum of
// squares is taken in their order (eight elements per lane, then the lanes by halves) and the norm's result is rounded to bf16 before it
// is rotated, so that the router of a mixture-of-experts layer behind it chooses as before. It replaces contiguous copies of q and k, two
// norms, two copies back, two rotations and the append: nine launches of 2 to 4 us each in a decode step, about 390 us per layer at 5,600
// tokens of training (now 79 us). For a backward pass the heads in front of the norm and their 1 / rms leave as well.
__global__ void __launch_bounds__(256)
qk_norm_rope_kernel(__nv_bfloat16* __restrict__ qkv, long long ld, const int* __restrict__ pos, const float* __restrict__ cos_t,
                    const float* __restrict__ sin_t, const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk, float eps,
                    const long long* __restrict__ slot, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                    __nv_bfloat16* __restrict__ pre_q, __nv_bfloat16* __restrict__ pre_k, float* __restrict__ rstd_q,
                    float* __restrict__ rstd_k, int T, int nh, int nkv, int hd) {
  const int heads = nh + nkv + (slot != nullptr ? nkv : 0);
  const long long item = blockIdx.x * 8LL + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= static_cast<long long>(T) * heads) return;
  const long long t = item / heads;
  const int h = static_cast<int>(item - t * heads);
  const long long s = slot != nullptr ? slot[t] : -1;
  __nv_bfloat16* base = qkv + t * ld + static_cast<long long>(h) * hd;
  const int nv = hd >> 3, hv = nv >> 1;  // 16-byte pieces of a head and of its half: hd is a multiple of 16, at most 256
  const bool on = lane < nv;
  if (h >= nh + nkv) {  // a value head: only appended
    if (s >= 0 && on)
      reinterpret_cast<uint4*>(vc + (s * nkv + (h - nh - nkv)) * hd)[lane] = reinterpret_cast<const uint4*>(base)[lane];
    return;
  }
  const bool is_k = h >= nh;
  uint4 raw = make_uint4(0u, 0u, 0u, 0u), wraw = raw;
  if (on) {
    raw = reinterpret_cast<const uint4*>(base)[lane];
    wraw = reinterpret_cast<const uint4*>(is_k ? wk : wq)[lane];
  }
  float f[8], g[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&raw)[j]);
    const float2 b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&wraw)[j]);
    f[2 * j] = a.x; f[2 * j + 1] = a.y;
    g[2 * j] = b.x; g[2 * j + 1] = b.y;
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  ss = wsum(ss);
  const float rstd = rsqrtf(ss / hd + eps);
  const long long row = is_k ? t * nkv + (h - nh) : t * nh + h;
  __nv_bfloat16* pre = is_k ? pre_k : pre_q;
  if (pre != nullptr) {
    if (lane == 0) (is_k ? rstd_k : rstd_q)[row] = rstd;
    if (on) reinterpret_cast<uint4*>(pre + row * hd)[lane] = raw;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16(f[j] * rstd * g[j]));
  const bool low = lane < hv;
  const int partner = low ? lane + hv : lane - hv;
  float o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = __shfl_sync(0xffffffffu, f[j], on ? partner : lane);
  if (!on) return;
  const long long tab = static_cast<long long>(pos[t]) * (hd >> 1) + (low ? lane : lane - hv) * 8;
  uint4 out;
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const float2 c = *reinterpret_cast<const float2*>(cos_t + tab + j), sn = *reinterpret_cast<const float2*>(sin_t + tab + j);
    // a c - b s with the second product rounded, b c + a s with the first one: the bits of the separate kernels, to which a test holds it
    reinterpret_cast<__nv_bfloat162*>(&out)[j >> 1] =
        low ? __floats2bfloat162_rn(__fmaf_rn(f[j], c.x, -__fmul_rn(o[j], sn.x)), __fmaf_rn(f[j + 1], c.y, -__fmul_rn(o[j + 1], sn.y)))
            : __floats2bfloat162_rn(__fmaf_rn(o[j], sn.x, __fmul_rn(f[j], c.x)), __fmaf_rn(o[j + 1], sn.y, __fmul_rn(f[j + 1], c.y)));
  }
  reinterpret_cast<uint4*>(base)[lane] = out;
  if (is_k && s >= 0) reinterpret_cast<uint4*>(kc + (s * nkv + (h - nh)) * hd)[lane] = out;
}

// ------------------------------------------------------------------------------------------ decode attention
// q: [B, nh, hd] (row stride ldq); cache: [num_slots, nkv, hd]; block_table: [B, max_blocks]; ctx_len: [B].
// grid = (B, nkv); 4 warps; each warp walks 32-token tiles: the score phase is lane-per-token (no shuffles
// in the dot products), the value phase lane-per-dimension (coalesced 256-byte rows).
constexpr int DEC_WARPS = 4;
constexpr int MAXG = 8;

template <int HD>
__global__ void __launch_bounds__(DEC_WARPS * 32)
paged_decode_kernel(const __nv_bfloat16* __restrict__ q, long long ldq, const __nv_bfloat16* __restrict__ kc,
                    const __nv_bfloat16* __restrict__ vc, const int* __restrict__ block_table, int max_blocks,
                    const int* __restrict__ ctx_len, __nv_bfloat16* __restrict__ out, long long ldo, int nh, int nkv,
                    int block_size, float scale_log2) {
  constexpr int DPL = HD / 32;  // dims per lane in the value phase
  const int b = blockIdx.x, kvh = blockIdx.y;
  const int G = nh / nkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int len = ctx_len[b];

  __shared__ float q_s[MAXG][HD];
  __shared__ float p_s[DEC_WARPS][MAXG][32];
  __shared__ float o_s[DEC_WARPS][MAXG][HD];
  __shared__ float ml_s[DEC_WARPS][MAXG][2];

  for (int i = threadIdx.x; i < G * HD; i += blockDim.x) {
    const int g = i / HD, d = i % HD;
    q_s[g][d] = __bfloat162float(q[b * ldq + static_cast<long long>(kvh * G + g) * HD + d]) * scale_log2;
  }
  __syncthreads();

  float m[MAXG], l[MAXG], o[MAXG][DPL];
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int d = 0; d < DPL; ++d) o[g][d] = 0.f;
  }
  const int* bt = block_table + static_cast<long long>(b) * max_blocks;
  const long long row_stride = static_cast<long long>(nkv) * HD;

  for (int t0 = warp * 32; t0 < len; t0 += DEC_WARPS * 32) {
    const int t = t0 + lane;
    const bool valid = t < len;
    long long row = 0;
    if (valid) row = (static_cast<long long>(bt[t / block_size]) * block_size + (t % block_size)) * row_stride +
                     static_cast<long long>(kvh) * HD;
    float s[MAXG];
#pragma unroll
    for (int g = 0; g < MAXG; ++g) s[g] = 0.f;
    if (valid) {
      const uint4* kr = reinterpret_cast<const uint4*>(kc + row);
#pragma unroll 4
      for (int c = 0; c < HD / 8; ++c) {
        const uint4 kv = kr[c];
        const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&kv);
        float kf[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(k2[j]);
          kf[2 * j] = f.x;
          kf[2 * j + 1] = f.y;
        }
#pragma unroll
        for (int g = 0; g < MAXG; ++g) {
          if (g < G) {
            const float4 qa = *reinterpret_cast<const float4*>(&q_s[g][c * 8]);
            const float4 qb = *reinterpret_cast<const float4*>(&q_s[g][c * 8 + 4]);
            s[g] += qa.x * kf[0] + qa.y * kf[1] + qa.z * kf[2] + qa.w * kf[3] + qb.x * kf[4] + qb.y * kf[5] +
                    qb.z * kf[6] + qb.w * kf[7];
          }
        }
      }
    }
    float alpha[MAXG];
#pragma unroll
    for (int g = 0; g < MAXG; ++g) {
      if (g < G) {
        const float sv = valid ? s[g] : -INFINITY;
        const float mn = fmaxf(m[g], wmax(sv));
        const float p = exp2f(sv - mn);
        alpha[g] = exp2f(m[g] - mn);
        l[g] = l[g] * alpha[g] + wsum(p);
        m[g] = mn;
        p_s[warp][g][lane] = p;
      }
    }
    __syncwarp();
#pragma unroll
    for (int g = 0; g < MAXG; ++g) {
      if (g < G) {
#pragma unroll
        for (int d = 0; d < DPL; ++d) o[g][d] *= alpha[g];
      }
    }
    const int nt = min(32, len - t0);
    for (int tt = 0; tt < nt; ++tt) {
      const long long r = __shfl_sync(0xffffffffu, row, tt);
      float vf[DPL];
      if constexpr (DPL == 4) {
        const uint2 raw = *reinterpret_cast<const uint2*>(vc + r + lane * 4);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 c = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        vf[0] = a.x; vf[1] = a.y; vf[2] = c.x; vf[3] = c.y;
      } else {
        const uint32_t raw = *reinterpret_cast<const uint32_t*>(vc + r + lane * 2);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
        vf[0] = a.x; vf[1] = a.y;
      }
#pragma unroll
      for (int g = 0; g < MAXG; ++g) {
        if (g < G) {
          const float p = p_s[warp][g][tt];
#pragma unroll
          for (int d = 0; d < DPL; ++d) o[g][d] += p * vf[d];
        }
      }
    }
    __syncwarp();
  }

  // merge the four warps
#pragma unroll
  for (int g = 0; g < MAXG; ++g) {
    if (g < G) {
      if (lane == 0) {
        ml_s[warp][g][0] = m[g];
        ml_s[warp][g][1] = l[g];
      }
#pragma unroll
      for (int d = 0; d < DPL; ++d) o_s[warp][g][lane * DPL + d] = o[g][d];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < G * HD; i += blockDim.x) {
    const int g = i / HD, d = i % HD;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) M = fmaxf(M, ml_s[w][g][0]);
    float L = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float f = (ml_s[w][g][0] == -INFINITY) ? 0.f : exp2f(ml_s[w][g][0] - M);
      L += ml_s[w][g][1] * f;
      acc += o_s[w][g][d] * f;
    }
    out[b * ldo + static_cast<long long>(kvh * G + g) * HD + d] = __float2bfloat16(L > 0.f ? acc / L : 0.f);
  }
}

// ------------------------------------------------------------------------------------------ sampler
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Token and log-prob of every row of logits [B, V] bf16 (row stride ld). Columns >= valid_vocab are masked out.
// Greedy when inv_temp <= 0 (the log-prob is then reported at temperature 1), else Gumbel-max over x + g(u_i) with
// u_i = ((mix64(key + i) >> 40) + 0.5) / 2^24 and g(u) = -log(-log(u)).
//
// A row is spread over a cluster of CTAs whose partial results meet in distributed shared memory, so that few rows still use the whole
// chip and many rows end together (a CTA per row: 320 rows were two waves of 148 x 2). A thread takes 8 neighbouring logits
// at a time: one rescaling of the running sum and one exponential per logit. That exponential also decides which logits need their two
// logarithms at all: x + g(u) can beat the warp's best score s only if u >= exp(-exp(x - s)), and exp(-t) >= 1 - t, so a logit with
// u < 1 - t, t = e^(x - m) e^(m - s), cannot win. The bound is widened by 66 / 2^24 and by 2^-10 + 2^-21 |m| in the exponent of t, far above
// the rounding of its terms (scores as large as m carry 2^-24 |m| each) and of the logarithms, and the 64 uppermost values of u always
// count as candidates, so the token is the one that evaluating every logit gives (of equal scores the first). The exponent is the difference
// of two logits as stored, times the scale: with the scale folded into one fma against a rounded maximum, the largest logit's own term was
// not 1, and log-probs near 0 were off by up to 2^-22 |m| and sometimes positive. What is left is the 64-bit hash; loading a turn ahead and
// collecting the candidates of a turn in a mask were both slower.
// 320 x 152064 at temperature 1, captured: 140 us with a CTA per row -> 92 us; greedy, where the row is what counts: 92 -> 34 us (15 us for the
// bytes at the copy rate).
constexpr int SAMPLE_THREADS = 256;

struct SamplePart {
  float m, l, best, best_x;  // m: largest logit as stored; l: sum of e^((x - m) / temperature)
  int best_i;
};
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// it2: log2(e) / temperature
__device__ __forceinline__ void sample_fold(SamplePart& a, const SamplePart& b, float it2) {
  const float mn = fmaxf(a.m, b.m);
  a.l = (mn == -INFINITY) ? a.l + b.l : a.l * exp2_approx((a.m - mn) * it2) + b.l * exp2_approx((b.m - mn) * it2);
  a.m = mn;
  if (b.best > a.best || (b.best == a.best && b.best_i < a.best_i)) {
    a.best = b.best;
    a.best_i = b.best_i;
    a.best_x = b.best_x;
  }
}

// mix64(key + i) >> 40: the last step of mix64, z ^ (z >> 31), touches only the lowest of the upper 32 bits, which the shift drops
__device__ __forceinline__ uint32_t sample_bits(uint64_t key, int i) {
  uint64_t z = key + static_cast<uint64_t>(i) + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return static_cast<uint32_t>(z >> 40);
}
__device__ __forceinline__ float sample_score(float x, uint32_t h) {
  const float u = (static_cast<float>(h) + 0.5f) * (1.0f / 16777216.0f);  // (0,1)
  return x - __logf(-__logf(u));
}
// the largest value of a warp (not NaN), through the order-preserving map of floats to unsigned integers
__device__ __forceinline__ float warp_max(float v) {
  const uint32_t f = __float_as_uint(v);
  const uint32_t k = __reduce_max_sync(0xffffffffu, (f & 0x80000000u) ? ~f : (f | 0x80000000u));
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

template <bool VEC, bool GREEDY>
__global__ void __launch_bounds__(SAMPLE_THREADS, 6)
sample_kernel(const __nv_bfloat16* __restrict__ logits, long long ld, int valid_vocab, float inv_temp,
              const long long* __restrict__ seeds, long long step, long long* __restrict__ tokens, float* __restrict__ logprobs) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int parts = static_cast<int>(cluster.num_blocks()), part = static_cast<int>(cluster.block_rank());
  const int row = blockIdx.x / parts;
  constexpr float LOG2E = 1.4426950408889634f;
  const float it = GREEDY ? 1.f : inv_temp, it2 = it * LOG2E;
  const __nv_bfloat16* lr = logits + row * ld;
  const uint64_t key = mix64(static_cast<uint64_t>(seeds[row]) ^ (static_cast<uint64_t>(step) * 0xD1342543DE82EF95ull));
  SamplePart a{-INFINITY, 0.f, -INFINITY, 0.f, 0x7fffffff};
  float warp_best = -INFINITY;
  const int stride = parts * SAMPLE_THREADS * 8;
  const int lane = threadIdx.x & 31;
  // every lane of a warp makes the same number of turns (the loop holds warp-wide exchanges): the bound is the warp's first logit
  for (int w0 = (part * SAMPLE_THREADS + static_cast<int>(threadIdx.x) - lane) * 8; w0 < valid_vocab; w0 += stride) {
    const int i0 = w0 + lane * 8;
    float x[8];  // as stored: the temperature comes in with the exponential's scale, and where a logit is a candidate
    if (VEC && i0 + 8 <= valid_vocab) {
      const uint4 raw = *reinterpret_cast<const uint4*>(lr + i0);
      const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[2 * j] = __uint_as_float(u[j] << 16);
        x[2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = i0 + j < valid_vocab ? __bfloat162float(lr[i0 + j]) : -INFINITY;
    }
    float mx = x[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, x[j]);
    const float mn = fmaxf(a.m, mx);
    const float ref = mn == -INFINITY ? 0.f : mn;  // nothing but masked logits so far: their exponentials are 0
    float sum = a.l * exp2_approx((a.m - ref) * it2);
    if (!GREEDY && warp_best == -INFINITY) {
      // a first score to beat: every lane's largest logit
      int jm = 0;
#pragma unroll
      for (int j = 7; j >= 0; --j) jm = x[j] == mx ? j : jm;
      a.best = sample_score(mx * it, sample_bits(key, i0 + jm));
      if (!(a.best > -INFINITY)) a.best = -INFINITY;  // masked or NaN: nothing to beat yet
      else {
        a.best_i = i0 + jm;
        a.best_x = mx * it;
      }
      warp_best = warp_max(a.best);
    }
    const float rt = ref * it;
    const float t_scale = 8388608.f * __expf(rt - warp_best + fmaf(fabsf(rt), 4.76837158e-7f, 9.765625e-4f));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float e = exp2_approx((x[j] - ref) * it2);
      sum += e;
      if (GREEDY) {
        if (x[j] > a.best) {
          a.best = x[j];
          a.best_i = i0 + j;
          a.best_x = x[j];
        }
      } else {
        // h / 2 as a float without a conversion (those run at the rate of the exponentials): 2^23 + h / 2
        const float bound = fmaf(-e, t_scale, 16777216.f - 33.f);
        const uint32_t h = sample_bits(key, i0 + j);
        if (!(__uint_as_float(0x4B000000u | (h >> 1)) < bound)) {  // a NaN bound counts as a candidate
          const float score = sample_score(x[j] * it, h);
          // (a score of -inf is a masked logit, or a lane behind the vocabulary's end: it takes no token, also in a row without numbers)
          if (score > a.best || (score == a.best && i0 + j < a.best_i && score > -INFINITY)) {
            a.best = score;
            a.best_i = i0 + j;
            a.best_x = x[j] * it;
          }
        }
      }
    }
    a.m = mn;
    a.l = sum;
    if (!GREEDY) warp_best = warp_max(a.best);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const SamplePart b{__shfl_xor_sync(0xffffffffu, a.m, o), __shfl_xor_sync(0xffffffffu, a.l, o), __shfl_xor_sync(0xffffffffu, a.best, o),
                       __shfl_xor_sync(0xffffffffu, a.best_x, o), __shfl_xor_sync(0xffffffffu, a.best_i, o)};
    sample_fold(a, b, it2);
  }
  __shared__ SamplePart warp_part[SAMPLE_THREADS / 32];
  __shared__ SamplePart cta_part;
  if (lane == 0) warp_part[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < SAMPLE_THREADS / 32; ++k) sample_fold(a, warp_part[k], it2);
    cta_part = a;
  }
  cluster.sync();
  if (part == 0 && threadIdx.x == 0) {
    for (int k = 1; k < parts; ++k) sample_fold(a, *cluster.map_shared_rank(&cta_part, k), it2);
    tokens[row] = a.best_i == 0x7fffffff ? 0 : a.best_i;
    if (logprobs) logprobs[row] = a.m == -INFINITY ? __int_as_float(0x7fffffff) : a.best_x - (a.m * it + __logf(a.l));  // no token: NaN
  }
  cluster.sync();  // a CTA's shared memory is read by its cluster until here
}

// ---- top-k / top-p (nucleus) sampling without a sort.
// bf16 logits have at most 65536 distinct values, so the k-th largest value and the nucleus boundary are found exactly by
// two rounds of 256-bin histograms over an order-preserving 16-bit key (high byte, then low byte inside the boundary
// bin): counts for top-k, probability mass for top-p (evaluated on the distribution that top-k left, as the reference
// samplers do). Every element whose key is >= the boundary key is kept: elements that tie with the boundary value stay
// in. The token is then drawn by Gumbel-max among the kept ones and its log-prob is that of the renormalised
// distribution. One block per row; the row (V * 2 bytes) is re-read from L2 by each pass.
__device__ __forceinline__ unsigned int bf16_key(__nv_bfloat16 v) {
  const unsigned int u = __bfloat16_as_ushort(v);
  return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
}

__global__ void sample_topkp_kernel(const __nv_bfloat16* __restrict__ logits, long long ld, int valid_vocab, float inv_temp,
                                    int top_k, float top_p, const long long* __restrict__ seeds, long long step,
                                    long long* __restrict__ tokens, float* __restrict__ logprobs) {
  const int row = blockIdx.x;
  const __nv_bfloat16* lr = logits + row * ld;
  __shared__ int cnt[256];
  __shared__ float mass[256];
  __shared__ float red[32];
  __shared__ int sh_i[4];
  __shared__ float sh_f[4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto block_max = [&](float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = red[0];
      for (int k = 1; k < nw; ++k) t = fmaxf(t, red[k]);
      sh_f[0] = t;
    }
    __syncthreads();
    const float r = sh_f[0];
    __syncthreads();
    return r;
  };
  auto block_sum = [&](float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int k = 0; k < nw; ++k) t += red[k];   // fixed order
      sh_f[0] = t;
    }
    __syncthreads();
    const float r = sh_f[0];
    __syncthreads();
    return r;
  };
  // pass A: row maximum (of the temperature-scaled logits)
  float m = -INFINITY;
  for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) m = fmaxf(m, __bfloat162float(lr[i]) * inv_temp);
  m = block_max(m);
  unsigned int thr = 0;  // keep key >= thr
  if (top_k > 0 && top_k < valid_vocab) {
    // passes B, C: the key of the k-th largest element
    for (int b = threadIdx.x; b < 256; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) atomicAdd(&cnt[bf16_key(lr[i]) >> 8], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      int c = 0, b = 255;
      for (; b > 0; --b) {
        if (c + cnt[b] >= top_k) break;
        c += cnt[b];
      }
      sh_i[0] = b;
      sh_i[1] = c;  // elements strictly above bin b
    }
    __syncthreads();
    const int hb = sh_i[0], above = sh_i[1];
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) {
      const unsigned int k = bf16_key(lr[i]);
      if (static_cast<int>(k >> 8) == hb) atomicAdd(&cnt[k & 255u], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int c = above, b = 255;
      for (; b > 0; --b) {
        if (c + cnt[b] >= top_k) break;
        c += cnt[b];
      }
      sh_i[2] = (hb << 8) | b;
    }
    __syncthreads();
    thr = static_cast<unsigned int>(sh_i[2]);
    __syncthreads();
  }
  if (top_p < 1.f) {
    // passes D, E: the smallest set of the largest elements whose mass reaches top_p of what top-k kept
    for (int b = threadIdx.x; b < 256; b += blockDim.x) mass[b] = 0.f;
    __syncthreads();
    float z = 0.f;
    for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) {
      const unsigned int k = bf16_key(lr[i]);
      if (k >= thr) {
        const float e = __expf(__bfloat162float(lr[i]) * inv_temp - m);
        z += e;
        atomicAdd(&mass[k >> 8], e);
      }
    }
    z = block_sum(z);
    if (threadIdx.x == 0) {
      float c = 0.f;
      int b = 255;
      for (; b > 0; --b) {
        if (c + mass[b] >= top_p * z) break;
        c += mass[b];
      }
      sh_i[0] = b;
      sh_f[1] = c;
    }
    __syncthreads();
    const int hb = sh_i[0];
    const float above = sh_f[1];
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) mass[b] = 0.f;
    __syncthreads();
    for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) {
      const unsigned int k = bf16_key(lr[i]);
      if (k >= thr && static_cast<int>(k >> 8) == hb) atomicAdd(&mass[k & 255u], __expf(__bfloat162float(lr[i]) * inv_temp - m));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float c = above;
      int b = 255;
      for (; b > 0; --b) {
        if (c + mass[b] >= top_p * z) break;
        c += mass[b];
      }
      const unsigned int tp = (static_cast<unsigned int>(hb) << 8) | static_cast<unsigned int>(b);
      sh_i[2] = static_cast<int>(tp > thr ? tp : thr);
    }
    __syncthreads();
    thr = static_cast<unsigned int>(sh_i[2]);
    __syncthreads();
  }
  // pass F: Gumbel-max among the kept elements, normaliser of the kept set
  const uint64_t key = mix64(static_cast<uint64_t>(seeds[row]) ^ (static_cast<uint64_t>(step) * 0xD1342543DE82EF95ull));
  float l = 0.f, best = -INFINITY, best_x = 0.f;
  int best_i = 0;
  for (int i = threadIdx.x; i < valid_vocab; i += blockDim.x) {
    if (bf16_key(lr[i]) < thr) continue;
    const float x = __bfloat162float(lr[i]) * inv_temp;
    l += __expf(x - m);
    const uint64_t h = mix64(key + static_cast<uint64_t>(i));
    const float u = (static_cast<float>(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
    const float score = x - __logf(-__logf(u));
    if (score > best) {
      best = score;
      best_i = i;
      best_x = x;
    }
  }
  l = block_sum(l);
  __shared__ float sb[32], sx[32];
  __shared__ int si[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float b2 = __shfl_xor_sync(0xffffffffu, best, o), x2 = __shfl_xor_sync(0xffffffffu, best_x, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (b2 > best || (b2 == best && i2 < best_i)) {
      best = b2;
      best_i = i2;
      best_x = x2;
    }
  }
  if (lane == 0) {
    sb[w] = best; sx[w] = best_x; si[w] = best_i;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nw; ++k) {
      if (sb[k] > best || (sb[k] == best && si[k] < best_i)) {
        best = sb[k];
        best_i = si[k];
        best_x = sx[k];
      }
    }
    tokens[row] = best_i;
    if (logprobs) logprobs[row] = best_x - (m + __logf(l));
  }
}

}  // namespace vb

using namespace vb;

extern "C" {

int vb_kv_append(const void* k, const void* v, long long ldk, long long ldv, const long long* slot, void* kc, void* vc,
                 int T, int nkv, int hd, cudaStream_t s) {
  if (T == 0) return 0;
  if ((nkv * hd) % 8) return -1;
  kv_append_kernel<<<T, 128, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(k), reinterpret_cast<const __nv_bfloat16*>(v),
                                     ldk, ldv, slot, reinterpret_cast<__nv_bfloat16*>(kc),
                                     reinterpret_cast<__nv_bfloat16*>(vc), nkv * hd);
  return static_cast<int>(cudaGetLastError());
}

int vb_rope_kv_append(void* qkv, long long ld, const int* pos, const float* cos_t, const float* sin_t, const long long* slot,
                      void* kc, void* vc, int T, int nh, int nkv, int hd, cudaStream_t s) {
  if (T == 0) return 0;
  if ((hd % 8) || (ld % 8) || ((nkv * hd) % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(vc)) & 15) return -2;
  rope_kv_append_kernel<<<T, 256, 0, s>>>(reinterpret_cast<__nv_bfloat16*>(qkv), ld, pos, cos_t, sin_t, slot,
                                          reinterpret_cast<__nv_bfloat16*>(kc), reinterpret_cast<__nv_bfloat16*>(vc), nh, nkv, hd);
  return static_cast<int>(cudaGetLastError());
}

// slot (with kc, vc) and the four pre_* / rstd_* outputs are optional
int vb_qk_norm_rope(void* qkv, long long ld, const int* pos, const float* cos_t, const float* sin_t, const void* wq, const void* wk, float eps,
                    const long long* slot, void* kc, void* vc, void* pre_q, void* pre_k, float* rstd_q, float* rstd_k, int T, int nh, int nkv,
                    int hd, cudaStream_t s) {
  if (T == 0) return 0;
  if ((hd % 16) || hd > 256 || (ld % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(wk) | reinterpret_cast<uintptr_t>(kc) |
       reinterpret_cast<uintptr_t>(vc)) & 15)
    return -2;
  if ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 7) return -2;
  const long long blocks = (static_cast<long long>(T) * (nh + nkv + (slot != nullptr ? nkv : 0)) + 7) / 8;
  if (blocks > 0x7fffffffLL) return -4;
  auto bf = [](const void* p) { return reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(p)); };
  qk_norm_rope_kernel<<<static_cast<int>(blocks), 256, 0, s>>>(bf(qkv), ld, pos, cos_t, sin_t, bf(wq), bf(wk), eps, slot, bf(kc), bf(vc), bf(pre_q),
                                                               bf(pre_k), rstd_q, rstd_k, T, nh, nkv, hd);
  return static_cast<int>(cudaGetLastError());
}

int vb_paged_decode(const void* q, long long ldq, const void* kc, const void* vc, const int* block_table,
                    int max_blocks, const int* ctx_len, void* out, long long ldo, int B, int nh, int nkv, int hd,
                    int block_size, float scale, cudaStream_t s) {
  if (B == 0) return 0;
  if (nh % nkv || nh / nkv > MAXG) return -1;
  const float sl2 = scale * 1.4426950408889634f;
  dim3 grid(B, nkv);
  if (hd == 128)
    paged_decode_kernel<128><<<grid, DEC_WARPS * 32, 0, s>>>(
        reinterpret_cast<const __nv_bfloat16*>(q), ldq, reinterpret_cast<const __nv_bfloat16*>(kc),
        reinterpret_cast<const __nv_bfloat16*>(vc), block_table, max_blocks, ctx_len,
        reinterpret_cast<__nv_bfloat16*>(out), ldo, nh, nkv, block_size, sl2);
  else if (hd == 64)
    paged_decode_kernel<64><<<grid, DEC_WARPS * 32, 0, s>>>(
        reinterpret_cast<const __nv_bfloat16*>(q), ldq, reinterpret_cast<const __nv_bfloat16*>(kc),
        reinterpret_cast<const __nv_bfloat16*>(vc), block_table, max_blocks, ctx_len,
        reinterpret_cast<__nv_bfloat16*>(out), ldo, nh, nkv, block_size, sl2);
  else
    return -2;
  return static_cast<int>(cudaGetLastError());
}

int vb_sample_topkp(const void* logits, long long ld, int B, int V, int valid_vocab, float inv_temp, int top_k, float top_p,
                    const long long* seeds, long long step, long long* tokens, float* logprobs, cudaStream_t s) {
  if (B == 0) return 0;
  if (valid_vocab <= 0 || valid_vocab > V) valid_vocab = V;
  if (inv_temp <= 0.f || top_p <= 0.f) return -1;  // greedy decoding goes through vb_sample
  sample_topkp_kernel<<<B, 1024, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(logits), ld, valid_vocab, inv_temp, top_k, top_p,
                                         seeds, step, tokens, logprobs);
  return static_cast<int>(cudaGetLastError());
}

int vb_sample(const void* logits, long long ld, int B, int V, int valid_vocab, float inv_temp, const long long* seeds,
              long long step, long long* tokens, float* logprobs, cudaStream_t s) {
  if (B == 0) return 0;
  if (valid_vocab <= 0 || valid_vocab > V) valid_vocab = V;
  // 16-byte loads where every row starts on a 16-byte boundary. CTAs per row: doubled up to the portable cluster size while every CTA has a
  // full turn of logits and the launch less than 16 CTAs per SM. (An SM holds six: at most 32 per SM come out of it, so that many rows still
  // end together, and 320 rows of 152064 get eight CTAs each.)
  const bool vec = reinterpret_cast<uintptr_t>(logits) % 16 == 0 && ld % 8 == 0;
  int parts = 1;
  while (parts < 8 && parts * SAMPLE_THREADS * 8 < valid_vocab && static_cast<long long>(B) * parts < 16LL * num_sms()) parts *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(B) * parts);
  cfg.blockDim = dim3(SAMPLE_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = parts;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const auto kernel = inv_temp <= 0.f ? (vec ? sample_kernel<true, true> : sample_kernel<false, true>)
                                      : (vec ? sample_kernel<true, false> : sample_kernel<false, false>);
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const __nv_bfloat16*>(logits), ld, valid_vocab, inv_temp, seeds,
                                             step, tokens, logprobs));
}

}  // extern "C"
