// Memory-bound fused kernels (bf16 activations, fp32 statistics): RMSNorm (+residual) fwd/bwd, RoPE,
// SwiGLU fwd/bwd, embedding fwd/bwd, fused AdamW (fp32 master -> bf16 working copy), gradient norm /
// clip coefficient, casts.  All use 16-byte vector accesses; every row length must be a multiple of 8.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace vb {

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; every thread receives the result. `red` must hold >= 32 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (lane < nw) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

// ------------------------------------------------------------------------------------------ RMSNorm
// y = x_eff * rstd * w, x_eff = x (+ residual); when residual != null, x_eff is written to res_out.
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int H,
                                   float eps) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * H);
  const bf16x8* rr = residual ? reinterpret_cast<const bf16x8*>(residual + row * H) : nullptr;
  bf16x8* ro = res_out ? reinterpret_cast<bf16x8*>(res_out + row * H) : nullptr;
  const int nv = H >> 3;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8];
    unpack8(xr[i], f);
    if (rr) {
      float g[8];
      unpack8(rr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      bf16x8 h = pack8(f);
      ro[i] = h;
      unpack8(h, f);  // statistics on the rounded residual stream, as the next reader sees it
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  const bf16x8* src = rr ? reinterpret_cast<const bf16x8*>(res_out + row * H) : xr;
  const bf16x8* wv = reinterpret_cast<const bf16x8*>(w);
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * H);
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8], g[8];
    unpack8(src[i], f);
    unpack8(wv[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
    yr[i] = pack8(f);
  }
}

// The same for many rows of at most 4096: a warp per row that keeps the row in registers, so nothing is read twice and no barrier is met.
// The sums are those of the kernel above to the bit, because a router behind a norm turns a changed last bit into another choice of
// experts: NW = 4 or 8 (the warps it has) partial sums per lane, each over every NW-th piece of 32 x 16 bytes, halved lane by lane
// (16, 8, 4, 2, 1) and then warp by warp (4, 2, 1); the halving steps exchange the partial sums they do not keep, 12 shuffles in place
// of 43. With residual, 16,000 rows of 896 / 2048 / 3584: 28.1 -> 22.8, 59.2 -> 48.7, 98.8 -> 92.1 us (5.0, 5.4, 5.0 TB/s).
template <int J, int NW>
__global__ void __launch_bounds__(128)
rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual, const __nv_bfloat16* __restrict__ w,
                        __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int T, int H,
                        float eps) {
  const long long row = blockIdx.x * static_cast<long long>(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= T) return;
  const int lane = threadIdx.x & 31, nv = H >> 3;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * H);
  const bf16x8* wv = reinterpret_cast<const bf16x8*>(w);
  bf16x8 v[J], g[J];  // g: first the residual, then the weight; every load of an array is issued before the first is used
#pragma unroll
  for (int j = 0; j < J; ++j)
    if (j * 32 + lane < nv) v[j] = xr[j * 32 + lane];
  if (residual != nullptr) {
    const bf16x8* rr = reinterpret_cast<const bf16x8*>(residual + row * H);
    bf16x8* ro = reinterpret_cast<bf16x8*>(res_out + row * H);
#pragma unroll
    for (int j = 0; j < J; ++j)
      if (j * 32 + lane < nv) g[j] = rr[j * 32 + lane];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      float a[8], b[8];
      unpack8(v[j], a);
      unpack8(g[j], b);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] += b[i];
      v[j] = pack8(a);
    }
#pragma unroll
    for (int j = 0; j < J; ++j)
      if (j * 32 + lane < nv) ro[j * 32 + lane] = v[j];
  }
#pragma unroll
  for (int j = 0; j < J; ++j)
    if (j * 32 + lane < nv) g[j] = wv[j * 32 + lane];
  float p[NW];
#pragma unroll
  for (int k = 0; k < NW; ++k) p[k] = 0.f;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    if (j * 32 + lane < nv) {
      float a[8];
      unpack8(v[j], a);
#pragma unroll
      for (int i = 0; i < 8; ++i) p[j % NW] += a[i] * a[i];
    }
  }
  // lanes 16 and 8 (and 4) apart: each keeps half of the partial sums
#pragma unroll
  for (int n = NW / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const float other = __shfl_xor_sync(0xffffffffu, up ? p[k] : p[n + k], o);
      p[k] = (up ? p[n + k] : p[k]) + other;
    }
  }
  float ss = p[0];
#pragma unroll
  for (int o = 16 / NW; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
#pragma unroll
  for (int o = 16; o >= 32 / NW; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rstd = rsqrtf(ss / H + eps);
  if (lane == 0 && rstd_out) rstd_out[row] = rstd;
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * H);
#pragma unroll
  for (int j = 0; j < J; ++j) {
    if (j * 32 + lane < nv) {
      float a[8], b[8];
      unpack8(v[j], a);
      unpack8(g[j], b);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = a[i] * rstd * b[i];
      yr[j * 32 + lane] = pack8(a);
    }
  }
}

// dx = rstd * (dy*w) - x * rstd^3 * mean(dy*w*x) (+ dres_in);  dw partial per block -> scratch[grid, H].
// A block walks over groups of RB rows; each thread owns fixed column vectors so the dw partial stays in registers
// (H <= 8 * VPT * blockDim.x). The rows of a group are loaded together and share one exchange over the block, which alternates between
// two buffers and so needs one barrier: with a row and two barriers at a time the block waited for memory once per row. With the fold of
// the partial sums, 16,000 rows of 896 / 3584: 58.4 -> 36.0, 165.5 -> 134.9 us.
template <int VPT, int RB>
__global__ void rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                   const __nv_bfloat16* __restrict__ dres_in, __nv_bfloat16* __restrict__ dx,
                                   float* __restrict__ dw_partial, int T, int H) {
  __shared__ float red[2][RB][8];
  const int nv = H >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;  // at most 8
  float dwacc[VPT][8];
  bf16x8 wreg[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = threadIdx.x + v * blockDim.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[v][j] = 0.f;
    if (i < nv) wreg[v] = reinterpret_cast<const bf16x8*>(w)[i];
  }
  int buf = 0;
  for (long long row0 = static_cast<long long>(blockIdx.x) * RB; row0 < T; row0 += static_cast<long long>(gridDim.x) * RB, buf ^= 1) {
    bf16x8 dyv[RB][VPT], xv[RB][VPT], dr[RB][VPT];
    float rs[RB], dot[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const long long row = min(row0 + r, static_cast<long long>(T) - 1);  // rows past the end repeat the last one and count nothing
      rs[r] = rstd[row];
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int i = threadIdx.x + v * blockDim.x;
        if (i < nv) {
          dyv[r][v] = reinterpret_cast<const bf16x8*>(dy + row * H)[i];
          xv[r][v] = reinterpret_cast<const bf16x8*>(x + row * H)[i];
          if (dres_in != nullptr) dr[r][v] = reinterpret_cast<const bf16x8*>(dres_in + row * H)[i];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      dot[r] = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        if (static_cast<int>(threadIdx.x + v * blockDim.x) < nv) {
          float a[8], b[8], c[8];
          unpack8(dyv[r][v], a);
          unpack8(xv[r][v], b);
          unpack8(wreg[v], c);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            dot[r] += a[j] * c[j] * b[j];
            if (row0 + r < T) dwacc[v][j] += a[j] * b[j] * rs[r];
          }
        }
      }
      dot[r] = warp_sum(dot[r]);
      if (lane == 0) red[buf][r][warp] = dot[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      if (row0 + r >= T) break;
      float d = 0.f;
      for (int k = 0; k < warps; ++k) d += red[buf][r][k];
      const float c = d * rs[r] * rs[r] * rs[r] / H;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int i = threadIdx.x + v * blockDim.x;
        if (i < nv) {
          float a[8], b[8], g[8], o[8];
          unpack8(dyv[r][v], a);
          unpack8(xv[r][v], b);
          unpack8(wreg[v], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = rs[r] * a[j] * g[j] - b[j] * c;
          if (dres_in != nullptr) {
            unpack8(dr[r][v], a);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += a[j];
          }
          reinterpret_cast<bf16x8*>(dx + (row0 + r) * H)[i] = pack8(o);
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = threadIdx.x + v * blockDim.x;
    if (i < nv) {
      float* dst = dw_partial + static_cast<long long>(blockIdx.x) * H + i * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(dwacc[v][0], dwacc[v][1], dwacc[v][2], dwacc[v][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(dwacc[v][4], dwacc[v][5], dwacc[v][6], dwacc[v][7]);
    }
  }
}

// dw[h] (+)= sum_b partial[b, h]: 32 columns per block, every warp an eighth of the rows, folded in a fixed order: 7 us for 592 rows of
// 896. (A thread per column walked all rows one after the other on four blocks: 24 us.)
__global__ void __launch_bounds__(256)
colsum_kernel(const float* __restrict__ partial, float* __restrict__ out, int B, int H, int accumulate) {
  __shared__ float part[8][33];
  const int h = blockIdx.x * 32 + (threadIdx.x & 31), warp = threadIdx.x >> 5;
  float s = 0.f;
  if (h < H) {
#pragma unroll 8
    for (int b = warp; b < B; b += 8) s += partial[static_cast<long long>(b) * H + h];
  }
  part[warp][threadIdx.x & 31] = s;
  __syncthreads();
  if (warp != 0 || h >= H) return;
  s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += part[k][threadIdx.x];
  out[h] = accumulate ? out[h] + s : s;
}

// Backward of the norms of the q and k heads, in place in the gradient of the projection [T, (nh + 2 nkv) * hd]. L lanes hold a head
// (16 bytes each), a group of them takes RB heads at a time; the partial sums of the weights' gradients leave per block,
// partial[0] q, partial[1] k, each [gridDim.x, hd]. In place it needs no copies of q and k to contiguous rows and back: 63 us now, with
// the copies and a block per head 335 + 126 us for the q heads alone (8 sequences, 32 + 4 heads of 128).
template <int L>
__global__ void __launch_bounds__(256)
qk_norm_bwd_kernel(__nv_bfloat16* __restrict__ g_qkv, long long ld, const __nv_bfloat16* __restrict__ pre_q,
                   const __nv_bfloat16* __restrict__ pre_k, const float* __restrict__ rstd_q, const float* __restrict__ rstd_k,
                   const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk, float* __restrict__ partial, int T, int nh,
                   int nkv, int hd) {
  constexpr int GROUPS = 256 / L, RB = 4;
  __shared__ float s_dw[GROUPS][8 * L + 4];
  const int l = threadIdx.x % L, group = threadIdx.x / L;
  const bool on = l < (hd >> 3);
  for (int kind = 0; kind < 2; ++kind) {
    const int heads = kind ? nkv : nh;
    const __nv_bfloat16* pre = kind ? pre_k : pre_q;
    const float* rstd = kind ? rstd_k : rstd_q;
    float wv[8], dw[8];
    bf16x8 raw{};
    if (on) raw = reinterpret_cast<const bf16x8*>(kind ? wk : wq)[l];
    unpack8(raw, wv);
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[j] = 0.f;
    const long long items = static_cast<long long>(T) * heads;
    const long long stride = static_cast<long long>(gridDim.x) * GROUPS * RB;
    // every lane of a warp makes the same number of turns: the bound is the block's first item
    for (long long base = static_cast<long long>(blockIdx.x) * GROUPS * RB; base < items; base += stride) {
      bf16x8 dy[RB], x[RB];
      float rs[RB];
      bf16x8* at[RB];
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const long long it = base + static_cast<long long>(r) * GROUPS + group;
        const bool ok = it < items;
        const long long t = ok ? it / heads : 0;
        const int h = ok ? static_cast<int>(it - t * heads) : 0;
        at[r] = reinterpret_cast<bf16x8*>(g_qkv + t * ld + static_cast<long long>(kind ? nh + h : h) * hd) + l;
        dy[r] = bf16x8{};
        x[r] = bf16x8{};
        rs[r] = ok ? rstd[it] : 0.f;
        if (ok && on) {
          dy[r] = *at[r];
          x[r] = reinterpret_cast<const bf16x8*>(pre + it * hd)[l];
        }
      }
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        float a[8], b[8], dot = 0.f;
        unpack8(dy[r], a);
        unpack8(x[r], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot += a[j] * wv[j] * b[j];
          dw[j] += a[j] * b[j] * rs[r];
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float c = dot * rs[r] * rs[r] * rs[r] / hd;
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = rs[r] * a[j] * wv[j] - b[j] * c;
        if (on && base + static_cast<long long>(r) * GROUPS + group < items) *at[r] = pack8(a);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s_dw[group][l * 8 + j] = dw[j];
    __syncthreads();
    for (int i = threadIdx.x; i < hd; i += 256) {
      float s = 0.f;
      for (int k = 0; k < GROUPS; ++k) s += s_dw[k][i];
      partial[(static_cast<long long>(kind) * gridDim.x + blockIdx.x) * hd + i] = s;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------ RoPE
// In place on x [T, nheads, hd] (row stride `ld` elements): HF rotate-half convention with a
// cos/sin table [max_pos, hd/2] (fp32).  sign = +1 forward, -1 backward (transpose of the rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t, int T, int nheads,
                            int hd, long long ld, float sign) {
  const int half = hd >> 1;
  const long long total = static_cast<long long>(T) * nheads * (half >> 1);  // two pairs per thread
  const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (idx >= total) return;
  const int pairs = half >> 1;
  const int i2 = static_cast<int>(idx % pairs);
  const int h = static_cast<int>((idx / pairs) % nheads);
  const long long t = idx / (static_cast<long long>(pairs) * nheads);
  const int p = pos[t];
  const int i = i2 * 2;
  __nv_bfloat16* base = x + t * ld + static_cast<long long>(h) * hd;
  const float2 c = *reinterpret_cast<const float2*>(cos_t + static_cast<long long>(p) * half + i);
  float2 s = *reinterpret_cast<const float2*>(sin_t + static_cast<long long>(p) * half + i);
  s.x *= sign;
  s.y *= sign;
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(base + i));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(base + half + i));
  *reinterpret_cast<__nv_bfloat162*>(base + i) = __floats2bfloat162_rn(a.x * c.x - b.x * s.x, a.y * c.y - b.y * s.y);
  *reinterpret_cast<__nv_bfloat162*>(base + half + i) =
      __floats2bfloat162_rn(b.x * c.x + a.x * s.x, b.y * c.y + a.y * s.y);
}

// ------------------------------------------------------------------------------------------ column sums
// Gradient of a bias: sums over the rows of a bf16 matrix. A block sums COLSUM_ROWS rows of 512 columns (two neighbouring columns per
// thread, 128 bytes per warp and row, eight rows in flight) into a plane of partial sums, a second launch folds the planes in order. A thread's
// rows go to eight sums that are added pair by pair, and the planes are folded in double: one chain over the rows and one over the planes left
// errors of 5e-8 to 9e-8 of the sum of magnitudes, where casting to fp32 and reducing that leaves 1.5e-8 to 2e-8; now 1e-8.
// 7,900 x 4608 in 15 us, 16,000 x 5120 in 44 us; the cast and the reduction took 138 and 290.
constexpr int COLSUM_ROWS = 64;
__device__ __forceinline__ float colsum_pairs(const float (&s)[8]) { return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7])); }
__global__ void __launch_bounds__(256)
colsum_part_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, int T, int N, float* __restrict__ part) {
  const int c = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (c >= N) return;
  const int t0 = blockIdx.y * COLSUM_ROWS, t1 = min(T, t0 + COLSUM_ROWS);
  float a[8], b[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) a[u] = b[u] = 0.f;
  const bool pair = c + 1 < N;
  const bool vec = pair && ldx % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0;
  int t = t0;
  if (vec) {
    for (; t + 8 <= t1; t += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + (t + u) * ldx + c));
        a[u] += v.x;
        b[u] += v.y;
      }
    }
  }
  for (; t < t1; t += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (t + u < t1) {
        a[u] += __bfloat162float(x[(t + u) * ldx + c]);
        if (pair) b[u] += __bfloat162float(x[(t + u) * ldx + c + 1]);
      }
    }
  }
  float* o = part + static_cast<long long>(blockIdx.y) * N + c;
  o[0] = colsum_pairs(a);
  if (pair) o[1] = colsum_pairs(b);
}
__global__ void __launch_bounds__(256)
colsum_fold_kernel(const float* __restrict__ part, int chunks, int N, float* __restrict__ out) {
  __shared__ double fold[8][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), warp = threadIdx.x >> 5;
  double s = 0.0;
  if (c < N) {
#pragma unroll 8
    for (int k = warp; k < chunks; k += 8) s += part[static_cast<long long>(k) * N + c];
  }
  fold[warp][threadIdx.x & 31] = s;
  __syncthreads();
  if (warp != 0 || c >= N) return;
  s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += fold[k][threadIdx.x];
  out[c] = static_cast<float>(out[c] + s);
}

// ------------------------------------------------------------------------------------------ SwiGLU
// gu [T, 2I]: gate = gu[:, :I], up = gu[:, I:].
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                  long long T, int I) {
  const int nv = I >> 3;
  const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (idx >= T * nv) return;
  const long long t = idx / nv;
  const int i = static_cast<int>(idx % nv);
  float g[8], u[8];
  unpack8(reinterpret_cast<const bf16x8*>(gu + t * 2 * I)[i], g);
  unpack8(reinterpret_cast<const bf16x8*>(gu + t * 2 * I + I)[i], u);
#pragma unroll
  for (int j = 0; j < 8; ++j) g[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  reinterpret_cast<bf16x8*>(out + t * I)[i] = pack8(g);
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, long long T, int I) {
  const int nv = I >> 3;
  const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (idx >= T * nv) return;
  const long long t = idx / nv;
  const int i = static_cast<int>(idx % nv);
  float g[8], u[8], d[8], dg[8], du[8];
  unpack8(reinterpret_cast<const bf16x8*>(gu + t * 2 * I)[i], g);
  unpack8(reinterpret_cast<const bf16x8*>(gu + t * 2 * I + I)[i], u);
  unpack8(reinterpret_cast<const bf16x8*>(dout + t * I)[i], d);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sg = 1.f / (1.f + __expf(-g[j]));
    du[j] = d[j] * g[j] * sg;
    dg[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
  }
  reinterpret_cast<bf16x8*>(dgu + t * 2 * I)[i] = pack8(dg);
  reinterpret_cast<bf16x8*>(dgu + t * 2 * I + I)[i] = pack8(du);
}

// ------------------------------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ w,
                                     __nv_bfloat16* __restrict__ out, int H, int V) {
  const long long t = blockIdx.x;
  long long id = ids[t];
  if (id < 0 || id >= V) id = 0;
  const bf16x8* src = reinterpret_cast<const bf16x8*>(w + id * H);
  bf16x8* dst = reinterpret_cast<bf16x8*>(out + t * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) dst[i] = src[i];
}
__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ dout,
                                     float* __restrict__ dw, int H, int V) {
  const long long t = blockIdx.x;
  const long long id = ids[t];
  if (id < 0 || id >= V) return;
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    atomicAdd(dw + id * H + i, __bfloat162float(dout[t * H + i]));
}

// ------------------------------------------------------------------------------------------ optimizer
// ctrl[0] = sum of squared gradients (accumulated by sumsq_kernel), ctrl[1] = clip coefficient,
// ctrl[2] = 1.0 when the step must be skipped (non-finite norm), ctrl[3] = grad norm.
constexpr int SUMSQ_MAX_BLOCKS = 148 * 8;
__device__ float g_sumsq_partial[SUMSQ_MAX_BLOCKS];  // scratch of the two-pass reduction (one call at a time per device)

__global__ void sumsq_kernel(const float* __restrict__ g, long long n, float* __restrict__ ctrl) {
  __shared__ float red[32];
  float s = 0.f;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long n4 = n >> 2;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4; i += stride) {
    const float4 v = reinterpret_cast<const float4*>(g)[i];
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  for (long long i = (n4 << 2) + blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n; i += stride)
    s += g[i] * g[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) g_sumsq_partial[blockIdx.x] = s;
}
// second pass: the block partials are folded in a fixed order (bitwise reproducible), then added to ctrl[0]
__global__ void sumsq_final_kernel(int blocks, float* __restrict__ ctrl) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < blocks; i += blockDim.x) s += g_sumsq_partial[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) ctrl[0] += s;
}
__global__ void clip_coef_kernel(float* __restrict__ ctrl, float max_norm) {
  const float norm = sqrtf(ctrl[0]);
  const bool finite = isfinite(norm);
  ctrl[3] = norm;
  ctrl[2] = finite ? 0.f : 1.f;
  ctrl[1] = (finite && max_norm > 0.f) ? fminf(1.f, max_norm / (norm + 1e-6f)) : 1.f;
}

// AdamW on a flat shard.  master (fp32) is updated in place; the bf16 working copy is refreshed in the
// same pass; the gradient is optionally zeroed for the next accumulation round.
struct AdamArgs {
  float lr, beta1, beta2, eps, wd, bc1, bc2_sqrt;
};
__device__ __forceinline__ void adamw_one(float& p, float g, float& m, float& v, const AdamArgs& a) {
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  p *= (1.f - a.lr * a.wd);
  const float denom = sqrtf(v) / a.bc2_sqrt + a.eps;
  p -= (a.lr / a.bc1) * (m / denom);
}
// 30 bytes an element. VEC: 4 elements a thread in 16-byte accesses (every pointer 16-byte aligned, the bf16 copy 8; the remainder of n
// goes to the last threads one by one): 2^28 elements back to back 1163 us (6.9 TB/s, a little above a plain copy's 6.5) instead of 1337 us with
// 4-byte accesses (6.0 TB/s).
template <bool VEC>
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ master, float* __restrict__ grad, float* __restrict__ m, float* __restrict__ v,
             __nv_bfloat16* __restrict__ out_bf16, long long n, const float* __restrict__ ctrl, AdamArgs a, float grad_scale, int zero_grad) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const bool skip = ctrl && ctrl[2] != 0.f;
  const float coef = (ctrl ? ctrl[1] : 1.f) * grad_scale;
  const long long n4 = VEC ? n >> 2 : 0;
  if (VEC && i < n4) {
    if (!skip) {
      const float4 g = reinterpret_cast<const float4*>(grad)[i];
      float4 p = reinterpret_cast<const float4*>(master)[i], mi = reinterpret_cast<const float4*>(m)[i], vi = reinterpret_cast<const float4*>(v)[i];
      adamw_one(p.x, g.x * coef, mi.x, vi.x, a);
      adamw_one(p.y, g.y * coef, mi.y, vi.y, a);
      adamw_one(p.z, g.z * coef, mi.z, vi.z, a);
      adamw_one(p.w, g.w * coef, mi.w, vi.w, a);
      reinterpret_cast<float4*>(m)[i] = mi;
      reinterpret_cast<float4*>(v)[i] = vi;
      reinterpret_cast<float4*>(master)[i] = p;
      if (out_bf16) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y), hi = __floats2bfloat162_rn(p.z, p.w);
        uint2 o;
        o.x = *reinterpret_cast<unsigned int*>(&lo);
        o.y = *reinterpret_cast<unsigned int*>(&hi);
        reinterpret_cast<uint2*>(out_bf16)[i] = o;
      }
    }
    if (zero_grad) reinterpret_cast<float4*>(grad)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const long long e = VEC ? (n4 << 2) + (i - n4) : i;
  if (e >= n) return;
  if (!skip) {
    float p = master[e], mi = m[e], vi = v[e];
    adamw_one(p, grad[e] * coef, mi, vi, a);
    m[e] = mi;
    v[e] = vi;
    master[e] = p;
    if (out_bf16) out_bf16[e] = __float2bfloat16(p);
  }
  if (zero_grad) grad[e] = 0.f;
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n,
                                     float scale) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(in[i] * scale);
}

// out_f32[i] (+)= bf16 in[i] * scale
__global__ void accum_bf16_f32_kernel(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, long long n,
                                      float scale, int accumulate) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i < n) {
    const float x = __bfloat162float(in[i]) * scale;
    out[i] = accumulate ? out[i] + x : x;
  }
}

}  // namespace vb

using namespace vb;

static inline int cdiv_ll(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

extern "C" {

int vb_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* res_out, float* rstd, int T,
                   int H, float eps, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8) return -1;
  // A warp per row where rows fill the chip. With fewer a block per row has the shorter chain of loads: with residual, 64 rows of 896 / 2048
  // / 3584 2.2, 2.4, 2.8 us against 2.3, 3.0, 4.4 us, 320 rows 2.5, 3.5, 4.4 against 2.6, 3.2, 4.8 us; 1,000 rows 3.5, 5.6, 8.7 against
  // 3.0, 4.3, 7.8 us. Rows of one piece per lane (heads of a norm) 1.9 against 2.1 us at 64 rows already.
  if (H <= 4096 && (T >= 640 || H <= 256)) {
    const int rows = T >= 1184 ? 4 : 1;  // few rows: a block each, so that they are spread over the chip
    const int pieces = (H / 8 + 31) / 32;
#define VB_RF(J, NW)                                                                                                                     \
  rmsnorm_fwd_warp_kernel<J, NW><<<(T + rows - 1) / rows, 32 * rows, 0, s>>>(                                                            \
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(residual), reinterpret_cast<const __nv_bfloat16*>(w), \
      reinterpret_cast<__nv_bfloat16*>(y), reinterpret_cast<__nv_bfloat16*>(res_out), rstd, T, H, eps)
    if (H < 2048) {
      if (pieces <= 1) VB_RF(1, 4);
      else if (pieces <= 4) VB_RF(4, 4);
      else VB_RF(8, 4);
    } else {
      if (pieces <= 8) VB_RF(8, 8);
      else VB_RF(16, 8);
    }
#undef VB_RF
    return static_cast<int>(cudaGetLastError());
  }
  const int threads = H >= 2048 ? 256 : 128;
  rmsnorm_fwd_kernel<<<T, threads, 0, s>>>(
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(residual),
      reinterpret_cast<const __nv_bfloat16*>(w), reinterpret_cast<__nv_bfloat16*>(y),
      reinterpret_cast<__nv_bfloat16*>(res_out), rstd, H, eps);
  return static_cast<int>(cudaGetLastError());
}

// Number of partial rows the backward writes: scratch must hold rmsnorm_bwd_blocks(T) * H floats.
int vb_rmsnorm_bwd_blocks(int T) {
  const int cap = 148 * 4;
  return T < cap ? (T > 0 ? T : 1) : cap;
}

int vb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres_in, void* dx,
                   float* dw, float* scratch, int T, int H, int accumulate_dw, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8) return -1;
  const int blocks = vb_rmsnorm_bwd_blocks(T);
  const int nv = H / 8;
  const int threads = nv <= 32 ? 32 : nv <= 64 ? 64 : nv <= 128 ? 128 : 256;
  const int vpt = (nv + threads - 1) / threads;
  const bool few = T <= 2 * blocks;  // one or two rows per block: no groups
#define VB_RB(V, RB)                                                                                           \
  rmsnorm_bwd_kernel<V, RB><<<blocks, threads, 0, s>>>(                                                             \
      reinterpret_cast<const __nv_bfloat16*>(dy), reinterpret_cast<const __nv_bfloat16*>(x),                   \
      reinterpret_cast<const __nv_bfloat16*>(w), rstd, reinterpret_cast<const __nv_bfloat16*>(dres_in),        \
      reinterpret_cast<__nv_bfloat16*>(dx), scratch, T, H)
  if (vpt <= 1 && few) VB_RB(1, 1);
  else if (vpt <= 1) VB_RB(1, 4);
  else if (vpt <= 2 && few) VB_RB(2, 1);
  else if (vpt <= 2) VB_RB(2, 4);
  else if (vpt <= 4) VB_RB(4, 1);
  else return -2;  // H > 8192
#undef VB_RB
  colsum_kernel<<<(H + 31) / 32, 256, 0, s>>>(scratch, dw, blocks, H, accumulate_dw);
  return static_cast<int>(cudaGetLastError());
}

// partial: 2 * vb_rmsnorm_bwd_blocks(T) * hd floats; dwq, dwk are added to
int vb_qk_norm_bwd(void* g_qkv, long long ld, const void* pre_q, const void* pre_k, const float* rstd_q, const float* rstd_k, const void* wq,
                   const void* wk, float* dwq, float* dwk, float* partial, int T, int nh, int nkv, int hd, cudaStream_t s) {
  if (T == 0) return 0;
  if ((hd % 8) || hd > 256 || (ld % 8)) return -1;
  for (const void* p : {static_cast<const void*>(g_qkv), pre_q, pre_k, wq, wk})
    if (reinterpret_cast<uintptr_t>(p) & 15) return -2;
  const int blocks = vb_rmsnorm_bwd_blocks(T);
  auto bf = [](const void* p) { return reinterpret_cast<const __nv_bfloat16*>(p); };
  auto* g = reinterpret_cast<__nv_bfloat16*>(g_qkv);
  if (hd <= 64) qk_norm_bwd_kernel<8><<<blocks, 256, 0, s>>>(g, ld, bf(pre_q), bf(pre_k), rstd_q, rstd_k, bf(wq), bf(wk), partial, T, nh, nkv, hd);
  else if (hd <= 128) qk_norm_bwd_kernel<16><<<blocks, 256, 0, s>>>(g, ld, bf(pre_q), bf(pre_k), rstd_q, rstd_k, bf(wq), bf(wk), partial, T, nh, nkv, hd);
  else qk_norm_bwd_kernel<32><<<blocks, 256, 0, s>>>(g, ld, bf(pre_q), bf(pre_k), rstd_q, rstd_k, bf(wq), bf(wk), partial, T, nh, nkv, hd);
  colsum_kernel<<<(hd + 31) / 32, 256, 0, s>>>(partial, dwq, blocks, hd, 1);
  colsum_kernel<<<(hd + 31) / 32, 256, 0, s>>>(partial + static_cast<long long>(blocks) * hd, dwk, blocks, hd, 1);
  return static_cast<int>(cudaGetLastError());
}

int vb_rope(void* x, const int* pos, const float* cos_t, const float* sin_t, int T, int nheads, int hd, long long ld,
            int backward, cudaStream_t s) {
  if (T == 0) return 0;
  if (hd % 4) return -1;
  const long long total = static_cast<long long>(T) * nheads * (hd / 4);
  rope_kernel<<<cdiv_ll(total, 256), 256, 0, s>>>(reinterpret_cast<__nv_bfloat16*>(x), pos, cos_t, sin_t, T, nheads,
                                                  hd, ld, backward ? -1.f : 1.f);
  return static_cast<int>(cudaGetLastError());
}

int vb_colsum_chunks(int T) { return (T + COLSUM_ROWS - 1) / COLSUM_ROWS; }
int vb_colsum_add(const void* x, long long ldx, int T, int N, float* part, float* out, cudaStream_t s) {
  const int chunks = vb_colsum_chunks(T);
  if (chunks > 65535) return -4;
  colsum_part_kernel<<<dim3((N + 511) / 512, chunks), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), ldx, T, N, part);
  colsum_fold_kernel<<<(N + 31) / 32, 256, 0, s>>>(part, chunks, N, out);
  return static_cast<int>(cudaGetLastError());
}

int vb_swiglu_fwd(const void* gu, void* out, long long T, int I, cudaStream_t s) {
  if (T == 0) return 0;
  if (I % 8) return -1;
  swiglu_fwd_kernel<<<cdiv_ll(T * (I / 8), 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(gu),
                                                            reinterpret_cast<__nv_bfloat16*>(out), T, I);
  return static_cast<int>(cudaGetLastError());
}
int vb_swiglu_bwd(const void* dout, const void* gu, void* dgu, long long T, int I, cudaStream_t s) {
  if (T == 0) return 0;
  if (I % 8) return -1;
  swiglu_bwd_kernel<<<cdiv_ll(T * (I / 8), 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(dout),
                                                            reinterpret_cast<const __nv_bfloat16*>(gu),
                                                            reinterpret_cast<__nv_bfloat16*>(dgu), T, I);
  return static_cast<int>(cudaGetLastError());
}

int vb_embedding_fwd(const long long* ids, const void* w, void* out, int T, int H, int V, cudaStream_t s) {
  if (T == 0) return 0;
  if (H % 8) return -1;
  embedding_fwd_kernel<<<T, 128, 0, s>>>(ids, reinterpret_cast<const __nv_bfloat16*>(w),
                                         reinterpret_cast<__nv_bfloat16*>(out), H, V);
  return static_cast<int>(cudaGetLastError());
}
int vb_embedding_bwd(const long long* ids, const void* dout, float* dw, int T, int H, int V, cudaStream_t s) {
  if (T == 0) return 0;
  embedding_bwd_kernel<<<T, 256, 0, s>>>(ids, reinterpret_cast<const __nv_bfloat16*>(dout), dw, H, V);
  return static_cast<int>(cudaGetLastError());
}

int vb_sumsq(const float* g, long long n, float* ctrl, cudaStream_t s) {
  if (n == 0) return 0;
  long long blocks = (n / 4 + 255) / 256;
  if (blocks > SUMSQ_MAX_BLOCKS) blocks = SUMSQ_MAX_BLOCKS;
  if (blocks < 1) blocks = 1;
  sumsq_kernel<<<static_cast<int>(blocks), 256, 0, s>>>(g, n, ctrl);
  sumsq_final_kernel<<<1, 256, 0, s>>>(static_cast<int>(blocks), ctrl);
  return static_cast<int>(cudaGetLastError());
}
int vb_clip_coef(float* ctrl, float max_norm, cudaStream_t s) {
  clip_coef_kernel<<<1, 1, 0, s>>>(ctrl, max_norm);
  return static_cast<int>(cudaGetLastError());
}
int vb_adamw(float* master, float* grad, float* m, float* v, void* out_bf16, long long n, const float* ctrl, float lr,
             float beta1, float beta2, float eps, float wd, int step, float grad_scale, int zero_grad,
             cudaStream_t s) {
  if (n == 0) return 0;
  const float bc1 = 1.f - powf(beta1, static_cast<float>(step));
  const float bc2s = sqrtf(1.f - powf(beta2, static_cast<float>(step)));
  const AdamArgs args{lr, beta1, beta2, eps, wd, bc1, bc2s};
  const uintptr_t at = reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(m) |
                       reinterpret_cast<uintptr_t>(v) | (reinterpret_cast<uintptr_t>(out_bf16) << 1);
  if (at % 16 == 0)
    adamw_kernel<true><<<cdiv_ll((n >> 2) + (n & 3), 256), 256, 0, s>>>(master, grad, m, v, reinterpret_cast<__nv_bfloat16*>(out_bf16), n,
                                                                       ctrl, args, grad_scale, zero_grad);
  else
    adamw_kernel<false><<<cdiv_ll(n, 256), 256, 0, s>>>(master, grad, m, v, reinterpret_cast<__nv_bfloat16*>(out_bf16), n, ctrl, args,
                                                        grad_scale, zero_grad);
  return static_cast<int>(cudaGetLastError());
}
int vb_cast_f32_bf16(const float* in, void* out, long long n, float scale, cudaStream_t s) {
  if (n == 0) return 0;
  cast_f32_bf16_kernel<<<cdiv_ll(n, 256), 256, 0, s>>>(in, reinterpret_cast<__nv_bfloat16*>(out), n, scale);
  return static_cast<int>(cudaGetLastError());
}
int vb_accum_bf16_f32(const void* in, float* out, long long n, float scale, int accumulate, cudaStream_t s) {
  if (n == 0) return 0;
  accum_bf16_f32_kernel<<<cdiv_ll(n, 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(in), out, n, scale,
                                                        accumulate);
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
