// Mixture-of-experts bookkeeping kernels: softmax + top-k router, row gather into the expert-grouped (128-row padded)
// layout, weighted combine back to token order, and the routing-weight gradient.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace vb {
int num_sms();

// One warp per token. logits [T, E] (bf16), E <= 1024. Writes the k largest softmax probabilities
// (optionally renormalised to sum 1), their expert ids, and bumps the per-expert histogram.
template <int MAX_PER_LANE>
__global__ void moe_route_topk_kernel(const __nv_bfloat16* __restrict__ logits, long long ld, int T, int E, int k, int renorm,
                                      float* __restrict__ weights, int* __restrict__ experts, int* __restrict__ counts) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T) return;
  const __nv_bfloat16* row = logits + static_cast<long long>(warp) * ld;
  float v[MAX_PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < MAX_PER_LANE; ++i) {
    const int e = lane + 32 * i;
    v[i] = e < E ? __bfloat162float(row[e]) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < MAX_PER_LANE; ++i) {
    v[i] = (lane + 32 * i < E) ? __expf(v[i] - mx) : -1.f;  // probabilities (unnormalised); -1 marks "taken / absent"
    sum += fmaxf(v[i], 0.f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
  float top_sum = 0.f;
  float my_w = 0.f;
  int my_e = 0;
  for (int j = 0; j < k; ++j) {
    float best = -1.f;
    int bi = 0;
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
      if (v[i] > best) { best = v[i]; bi = lane + 32 * i; }
    }
    // warp arg-max; ties go to the smaller expert id (as torch.topk on a sorted-stable backend does not guarantee an
    // order for exact ties, any fixed rule is acceptable)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
      if (lane + 32 * i == bi) v[i] = -1.f;
    }
    top_sum += best;
    if (lane == j) { my_w = best; my_e = bi; }
  }
  if (lane < k) {
    const float w = renorm ? my_w / top_sum : my_w * inv;
    weights[static_cast<long long>(warp) * k + lane] = w;
    experts[static_cast<long long>(warp) * k + lane] = my_e;
    atomicAdd(counts + my_e, 1);
  }
}

// dst[r, :] = src[map[r], :] * (scale ? scale[r] : 1), or zeros where map[r] < 0.   H % 8 == 0, 16-byte vectors.
// num_mtiles (or null): only the rows of the tiles in use are written; the buffer is sized for the worst case.
__global__ void moe_gather_rows_kernel(const __nv_bfloat16* __restrict__ src, long long lds, const int* __restrict__ map,
                                       const float* __restrict__ scale, __nv_bfloat16* __restrict__ dst, long long ldd,
                                       int rows, int H, const int* __restrict__ num_mtiles, int tile_rows) {
  const int vec = H >> 3;
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (num_mtiles != nullptr) rows = min(rows, *num_mtiles * tile_rows);
  if (i >= static_cast<long long>(rows) * vec) return;
  const int r = static_cast<int>(i / vec), c = static_cast<int>(i % vec) * 8;
  const int s = map[r];
  uint4 out = make_uint4(0u, 0u, 0u, 0u);
  if (s >= 0) {
    out = *reinterpret_cast<const uint4*>(src + static_cast<long long>(s) * lds + c);
    if (scale != nullptr) {
      const float f = scale[r];
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __bfloat1622float2(h[j]);
        h[j] = __floats2bfloat162_rn(t.x * f, t.y * f);
      }
    }
  }
  *reinterpret_cast<uint4*>(dst + static_cast<long long>(r) * ldd + c) = out;
}

// silu(gate) * up for the rows of the tiles in use; gu [rows, 2 I]
__global__ void __launch_bounds__(256)
moe_swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, int rows, int I,
                  const int* __restrict__ num_mtiles, int tile_rows) {
  const int vec = I >> 3;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  const int r = static_cast<int>(i / vec), c = static_cast<int>(i - static_cast<long long>(r) * vec) * 8;
  if (r >= min(rows, *num_mtiles * tile_rows)) return;
  const uint4 gv = *reinterpret_cast<const uint4*>(gu + static_cast<long long>(r) * 2 * I + c);
  const uint4 uv = *reinterpret_cast<const uint4*>(gu + static_cast<long long>(r) * 2 * I + I + c);
  const __nv_bfloat162 *hg = reinterpret_cast<const __nv_bfloat162*>(&gv), *hu = reinterpret_cast<const __nv_bfloat162*>(&uv);
  uint4 o;
  __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 g = __bfloat1622float2(hg[q]), u = __bfloat1622float2(hu[q]);
    ho[q] = __floats2bfloat162_rn(g.x / (1.f + __expf(-g.x)) * u.x, g.y / (1.f + __expf(-g.y)) * u.y);
  }
  *reinterpret_cast<uint4*>(out + static_cast<long long>(r) * I + c) = o;
}

// Expert-grouped row layout: every expert's rows start at a multiple of `tile` rows, in the order of the flat list of choices.
//   seg[e] first row of expert e (seg[E]: rows in use), tile_expert[i] expert of tile i, num_mtiles tiles in use,
//   slot[i] row of choice i, src[row] token of the row, -1 for padding.
// Short lists (moe_plan_kernel): one block per expert. Every block forms the prefix of the padded counts by itself, its warps count the
// expert's choices in their share of the list and then write them in list order, so the layout does not depend on the schedule. The list is
// read twice per expert from L2 instead of being sorted: one launch where the sort, the scans and the scatters took about twenty (80 us per
// layer for 256 choices). Time grows with experts x choices; long lists take the two launches below.
template <typename IT>
__global__ void __launch_bounds__(256)
moe_plan_kernel(const IT* __restrict__ experts, const int* __restrict__ counts, int n, int k, int E, int tile, int cap, int* __restrict__ slot,
                int* __restrict__ src, int* __restrict__ seg, int* __restrict__ tile_expert, int* __restrict__ num_mtiles) {
  __shared__ int s_warp[8];
  __shared__ int s_edge[3];  // first row of this block's expert, rows it has, rows in use
  __shared__ int s_hits[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.x;
  // prefix of the padded counts: thread t holds experts 4t .. 4t + 3
  int pad[4], sum = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int x = threadIdx.x * 4 + u;
    pad[u] = x < E ? (counts[x] + tile - 1) / tile * tile : 0;
    sum += pad[u];
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int first = incl - sum;
  for (int w = 0; w < warp; ++w) first += s_warp[w];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int x = threadIdx.x * 4 + u;
    if (x < E && e == 0) seg[x] = first;
    if (x == e) { s_edge[0] = first; s_edge[1] = pad[u]; }
    first += pad[u];
  }
  if (threadIdx.x == 255) {
    s_edge[2] = first;
    if (e == 0) { seg[E] = first; *num_mtiles = min(first, cap) / tile; }
  }
  __syncthreads();
  // counts that do not belong to the list cannot reach beyond the buffers
  const int row0 = min(s_edge[0], cap), rows = min(s_edge[1], cap - row0), used = s_edge[2];
  for (int i = threadIdx.x; i < rows / tile; i += 256) tile_expert[row0 / tile + i] = e;
  for (int i = used + e * 256 + threadIdx.x; i < cap; i += E * 256) src[i] = -1;
  for (int i = used / tile + e * 256 + threadIdx.x; i < cap / tile; i += E * 256) tile_expert[i] = E - 1;
  // choices of this expert in this warp's share of the list
  constexpr int U = 8;
  const int per = ((n + 7) / 8 + 31) / 32 * 32, lo = min(n, warp * per), hi = min(n, lo + per);
  int hits = 0;
  for (int i = lo; i < hi; i += 32 * U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int x = i + u * 32 + lane;
      hits += __popc(__ballot_sync(0xffffffffu, x < hi && static_cast<int>(experts[min(x, n - 1)]) == e));
    }
  }
  if (lane == 0) s_hits[warp] = hits;
  __syncthreads();
  int at = 0, total = 0;
  for (int w = 0; w < 8; ++w) {
    if (w < warp) at += s_hits[w];
    total += s_hits[w];
  }
  for (int i = total + threadIdx.x; i < rows; i += 256) src[row0 + i] = -1;
  for (int i = lo; i < hi; i += 32 * U) {
    bool mine[U];
    unsigned int bal[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int x = i + u * 32 + lane, id = static_cast<int>(experts[min(x, n - 1)]);
      mine[u] = x < hi && id == e;
      if (e == 0 && x < hi && (id < 0 || id >= E)) slot[x] = 0;  // no such expert: nothing behind it may be read out of range
      bal[u] = __ballot_sync(0xffffffffu, mine[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (mine[u]) {
        const int x = i + u * 32 + lane, j = at + __popc(bal[u] & ((1u << lane) - 1));
        slot[x] = j < rows ? row0 + j : 0;
        if (j < rows) src[row0 + j] = x / k;
      }
      at += __popc(bal[u]);
    }
  }
}

// The same layout for long lists: every block takes a piece of the list. The first launch counts a piece's choices per expert, the second
// places them: behind the earlier pieces' (their counts are summed up again by every block), the block's warps one behind the other, and
// within 32 choices by the rank among the lanes with the same expert. The list is read three times in all, whatever the number of experts:
// 65536 x 8 choices of 128 / 1024 experts 32 / 67 us, where one launch takes 510 / 733 and the sort took about 300.
template <typename IT>
__global__ void __launch_bounds__(256)
moe_plan_count_kernel(const IT* __restrict__ experts, int n, int per_block, int E, int* __restrict__ hist) {
  extern __shared__ int s_plan[];  // [E]
  for (int e = threadIdx.x; e < E; e += 256) s_plan[e] = 0;
  __syncthreads();
  const int lo = blockIdx.x * per_block, hi = min(n, lo + per_block);
  for (int i = lo + threadIdx.x; i < hi; i += 256) {
    const IT id = experts[i];
    if (id >= 0 && id < E) atomicAdd(s_plan + static_cast<int>(id), 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += 256) hist[static_cast<long long>(blockIdx.x) * E + e] = s_plan[e];
}

template <typename IT>
__global__ void __launch_bounds__(256)
moe_plan_place_kernel(const IT* __restrict__ experts, const int* __restrict__ counts, const int* __restrict__ hist, int n, int per_block, int k,
                      int E, int tile, int cap, int* __restrict__ slot, int* __restrict__ src, int* __restrict__ seg,
                      int* __restrict__ tile_expert, int* __restrict__ num_mtiles) {
  extern __shared__ int s_plan[];
  int* first = s_plan;          // [E + 1] first row of every expert
  int* at = s_plan + E + 1;     // [8][E] next row of a warp's choices
  __shared__ int s_warp[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, blk = blockIdx.x, blocks = gridDim.x;
  // prefix of the padded counts: thread t holds experts 4t .. 4t + 3
  int pad[4], sum = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int x = threadIdx.x * 4 + u;
    pad[u] = x < E ? (max(counts[x], 0) + tile - 1) / tile * tile : 0;
    sum += pad[u];
  }
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  for (int i = threadIdx.x; i < 8 * E; i += 256) at[i] = 0;
  __syncthreads();
  int row = incl - sum;
  for (int w = 0; w < warp; ++w) row += s_warp[w];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int x = threadIdx.x * 4 + u;
    if (x <= E) first[x] = row;
    row += pad[u];
  }
  if (threadIdx.x == 255 && E == 1024) first[E] = row;
  // choices per expert in every warp's share
  const int per = per_block / 8;  // a multiple of 32
  const int lo = min(n, blk * per_block + warp * per), hi = min(n, lo + per);
  int* mine = at + warp * E;
  for (int i = lo + lane; i < hi; i += 32) {
    const IT id = experts[i];
    if (id >= 0 && id < E) atomicAdd(mine + static_cast<int>(id), 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += 256) {
    int r = first[e];
#pragma unroll 8
    for (int c = 0; c < blk; ++c) r += hist[static_cast<long long>(c) * E + e];
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int v = at[w * E + e];
      at[w * E + e] = r;
      r += v;
    }
  }
  __syncthreads();
  for (int i = lo; i < hi; i += 32) {
    const int x = i + lane;
    const IT raw = x < hi ? experts[x] : IT(-1);
    const int id = raw >= 0 && raw < E ? static_cast<int>(raw) : -1;
    const unsigned int same = __match_any_sync(0xffffffffu, id);
    int pos = 0;
    if (id >= 0) pos = mine[id] + __popc(same & ((1u << lane) - 1));
    __syncwarp();
    if (id >= 0 && lane == 31 - __clz(same)) mine[id] = pos + 1;
    __syncwarp();
    if (x < hi) {
      // no such expert, or counts that do not belong to the list: nothing behind it may be read or written out of range
      const bool ok = id >= 0 && pos < min(first[id + 1], cap);
      slot[x] = ok ? pos : 0;
      if (ok) src[pos] = x / k;
    }
  }
  // padding rows and tiles: a warp per expert
  for (int e = blk * 8 + warp; e < E; e += blocks * 8) {
    int total = 0;
    for (int c = lane; c < blocks; c += 32) total += hist[static_cast<long long>(c) * E + e];
    total = __reduce_add_sync(0xffffffffu, total);
    const int row0 = min(first[e], cap), row1 = min(first[e + 1], cap);
    for (int i = row0 + min(total, row1 - row0) + lane; i < row1; i += 32) src[i] = -1;
    for (int i = row0 / tile + lane; i < row1 / tile; i += 32) tile_expert[i] = e;
  }
  const int used = first[E];
  for (int i = used + blk * 256 + threadIdx.x; i < cap; i += blocks * 256) src[i] = -1;
  for (int i = used / tile + blk * 256 + threadIdx.x; i < cap / tile; i += blocks * 256) tile_expert[i] = E - 1;
  if (blk == 0) {
    for (int e = threadIdx.x; e <= E; e += 256) seg[e] = first[e];
    if (threadIdx.x == 0) *num_mtiles = min(used, cap) / tile;
  }
}

// out[t, :] = sum_j w[t, j] * y[slot[t, j], :]   (fp32 accumulation in a fixed order: deterministic)
__global__ void moe_combine_kernel(const __nv_bfloat16* __restrict__ y, long long ldy, const int* __restrict__ slot,
                                   const float* __restrict__ w, __nv_bfloat16* __restrict__ out, long long ldo, int T, int H,
                                   int k) {
  const int vec = H >> 3;
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<long long>(T) * vec) return;
  const int t = static_cast<int>(i / vec), c = static_cast<int>(i % vec) * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // eight choices at a time: their rows are all on the way before the first is added
  for (int j0 = 0; j0 < k; j0 += 8) {
    uint4 v[8];
    float f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long long j = static_cast<long long>(t) * k + min(j0 + u, k - 1);
      f[u] = w != nullptr ? w[j] : 1.f;
      v[u] = *reinterpret_cast<const uint4*>(y + static_cast<long long>(slot[j]) * ldy + c);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (j0 + u >= k) break;
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[u]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 p2 = __bfloat1622float2(h[q]);
        acc[2 * q] += f[u] * p2.x;
        acc[2 * q + 1] += f[u] * p2.y;
      }
    }
  }
  uint4 o;
  __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int q = 0; q < 4; ++q) ho[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
  *reinterpret_cast<uint4*>(out + static_cast<long long>(t) * ldo + c) = o;
}

// gw[t, j] = <g[t, :], y[slot[t, j], :]>   one warp per (t, j)
__global__ void moe_combine_bwd_w_kernel(const __nv_bfloat16* __restrict__ g, long long ldg, const __nv_bfloat16* __restrict__ y,
                                         long long ldy, const int* __restrict__ slot, float* __restrict__ gw, int T, int H,
                                         int k) {
  const long long warp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= static_cast<long long>(T) * k) return;
  const int t = static_cast<int>(warp / k);
  const int s = slot[warp];
  const __nv_bfloat16* a = g + static_cast<long long>(t) * ldg;
  const __nv_bfloat16* b = y + static_cast<long long>(s) * ldy;
  float acc = 0.f;
  for (int c = lane * 8; c < H; c += 256) {
    const uint4 va = *reinterpret_cast<const uint4*>(a + c), vb_ = *reinterpret_cast<const uint4*>(b + c);
    const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&va);
    const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&vb_);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 x = __bfloat1622float2(ha[q]), z = __bfloat1622float2(hb[q]);
      acc += x.x * z.x + x.y * z.y;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) gw[warp] = acc;
}

// ---- expert parallelism over peer memory ------------------------------------------------------------------------
// Dispatch: the permutation into the expert-grouped layout writes each token copy straight into the buffer of the rank
// that owns the expert (peer stores over NVLink): permutation and all-to-all are one kernel, nothing is staged.
//   dst_ptrs[r] = base of rank r's grouped activation buffer [cap, H]; (dest_rank, dest_row) per (token, choice)
__global__ void moe_dispatch_peer_kernel(const __nv_bfloat16* __restrict__ src, long long lds, const unsigned long long* __restrict__ dst_ptrs,
                                         const int* __restrict__ dest_rank, const int* __restrict__ dest_row, int pairs, int k, int H) {
  const int vec = H >> 3;
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<long long>(pairs) * vec) return;
  const int pr = static_cast<int>(i / vec), c = static_cast<int>(i % vec) * 8;
  const int row = dest_row[pr];
  if (row < 0) return;  // dropped by the capacity limit
  const uint4 v = *reinterpret_cast<const uint4*>(src + static_cast<long long>(pr / k) * lds + c);
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(dst_ptrs[dest_rank[pr]]);
  *reinterpret_cast<uint4*>(dst + static_cast<long long>(row) * H + c) = v;
}

// Combine: out[t] = sum_j w[t,j] * y_{rank(t,j)}[row(t,j)] with the expert outputs read from the owners' buffers (peer
// loads): un-permutation, all-to-all and the weighted sum are one kernel.
__global__ void moe_combine_peer_kernel(const unsigned long long* __restrict__ y_ptrs, const int* __restrict__ src_rank,
                                        const int* __restrict__ src_row, const float* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                        long long ldo, int T, int H, int k) {
  const int vec = H >> 3;
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<long long>(T) * vec) return;
  const int t = static_cast<int>(i / vec), c = static_cast<int>(i % vec) * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int j = 0; j < k; ++j) {
    const long long pr = static_cast<long long>(t) * k + j;
    const int row = src_row[pr];
    if (row < 0) continue;
    const float f = w != nullptr ? w[pr] : 1.f;
    const __nv_bfloat16* y = reinterpret_cast<const __nv_bfloat16*>(y_ptrs[src_rank[pr]]);
    const uint4 v = *reinterpret_cast<const uint4*>(y + static_cast<long long>(row) * H + c);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 p2 = __bfloat1622float2(h[q]);
      acc[2 * q] += f * p2.x;
      acc[2 * q + 1] += f * p2.y;
    }
  }
  uint4 o;
  __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int q = 0; q < 4; ++q) ho[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
  *reinterpret_cast<uint4*>(out + static_cast<long long>(t) * ldo + c) = o;
}

// Every rank publishes its per-expert token counts into row `rank` of every peer's [W, E] table.
__global__ void moe_publish_counts_kernel(const int* __restrict__ counts, const unsigned long long* __restrict__ table_ptrs, int W,
                                          int rank, int E) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= W * E) return;
  const int r = i / E, e = i % E;
  reinterpret_cast<int*>(table_ptrs[r])[rank * E + e] = counts[e];
}

}  // namespace vb

using namespace vb;

extern "C" int vb_moe_dispatch_peer(const void* src, long long lds, const unsigned long long* dst_ptrs_dev, const int* dest_rank,
                                    const int* dest_row, int pairs, int k, int H, cudaStream_t s) {
  if (pairs <= 0) return 0;
  if (H % 8 || lds % 8) return -1;
  const long long n = static_cast<long long>(pairs) * (H / 8);
  moe_dispatch_peer_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(src), lds, dst_ptrs_dev,
                                                                             dest_rank, dest_row, pairs, k, H);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_combine_peer(const unsigned long long* y_ptrs_dev, const int* src_rank, const int* src_row, const float* w, void* out,
                                   long long ldo, int T, int H, int k, cudaStream_t s) {
  if (T <= 0) return 0;
  if (H % 8 || ldo % 8) return -1;
  const long long n = static_cast<long long>(T) * (H / 8);
  moe_combine_peer_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, s>>>(y_ptrs_dev, src_rank, src_row, w,
                                                                            reinterpret_cast<__nv_bfloat16*>(out), ldo, T, H, k);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_publish_counts(const int* counts, const unsigned long long* table_ptrs_dev, int W, int rank, int E, cudaStream_t s) {
  moe_publish_counts_kernel<<<(W * E + 255) / 256, 256, 0, s>>>(counts, table_ptrs_dev, W, rank, E);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_route_topk(const void* logits, long long ld, int T, int E, int k, int renorm, float* weights, int* experts,
                                 int* counts, cudaStream_t s) {
  if (T <= 0) return 0;
  if (E > 1024 || k > 32 || k > E) return -1;
  const int blocks = (T * 32 + 255) / 256;
  const auto* lg = reinterpret_cast<const __nv_bfloat16*>(logits);
  if (E <= 128) moe_route_topk_kernel<4><<<blocks, 256, 0, s>>>(lg, ld, T, E, k, renorm, weights, experts, counts);
  else if (E <= 256) moe_route_topk_kernel<8><<<blocks, 256, 0, s>>>(lg, ld, T, E, k, renorm, weights, experts, counts);
  else moe_route_topk_kernel<32><<<blocks, 256, 0, s>>>(lg, ld, T, E, k, renorm, weights, experts, counts);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_gather_rows(const void* src, long long lds, const int* map, const float* scale, void* dst, long long ldd,
                                  int rows, int H, const int* num_mtiles, int tile_rows, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (H % 8 || lds % 8 || ldd % 8) return -1;
  const long long n = static_cast<long long>(rows) * (H / 8);
  moe_gather_rows_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(src), lds, map, scale,
                                                                           reinterpret_cast<__nv_bfloat16*>(dst), ldd, rows, H, num_mtiles,
                                                                           tile_rows);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_swiglu(const void* gu, void* out, int rows, int I, const int* num_mtiles, int tile_rows, cudaStream_t s) {
  if (rows <= 0) return 0;
  if (I % 8) return -1;
  const long long n = static_cast<long long>(rows) * (I / 8);
  moe_swiglu_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(gu),
                                                                      reinterpret_cast<__nv_bfloat16*>(out), rows, I, num_mtiles, tile_rows);
  return static_cast<int>(cudaGetLastError());
}

// Up to here one launch is better: 8192 choices of 64 / 128 / 512 / 1024 experts 8 / 8.3 / 10.8 / 16.5 us against 8 / 9.0 / 15.4 / 24.8 with
// two; 16384 choices 13 / 13.2 / 17.5 / 27.2 against 8.4 / 9.3 / 13.8 / 22.5.
constexpr int PLAN_ONE_LAUNCH = 8192;
// A block per SM, in pieces of at least 1024 choices: every block sums up the counts of all pieces before its own.
static int plan_per_block(int n) {
  const int even = (n + num_sms() - 1) / num_sms();
  return even <= 1024 ? 1024 : (even + 255) / 256 * 256;
}
// Blocks of the two-launch form, 0 for one launch.
extern "C" int vb_moe_plan_blocks(int n) {
  if (n <= PLAN_ONE_LAUNCH) return 0;
  return (n + plan_per_block(n) - 1) / plan_per_block(n);
}

// experts: [n] int64 (wide) or int32; n = tokens * k choices. E <= 1024, cap a multiple of tile that holds every segment.
// hist: vb_moe_plan_blocks(n) * E integers.
template <typename IT>
static int moe_plan_launch(const IT* experts, const int* counts, int* hist, int n, int k, int E, int tile, int cap, int* slot, int* src, int* seg,
                           int* tile_expert, int* num_mtiles, cudaStream_t s) {
  const int blocks = vb_moe_plan_blocks(n);
  if (blocks == 0) {
    moe_plan_kernel<IT><<<E, 256, 0, s>>>(experts, counts, n, k, E, tile, cap, slot, src, seg, tile_expert, num_mtiles);
  } else {
    const int per = plan_per_block(n);
    moe_plan_count_kernel<IT><<<blocks, 256, E * sizeof(int), s>>>(experts, n, per, E, hist);
    moe_plan_place_kernel<IT><<<blocks, 256, (9 * E + 1) * sizeof(int), s>>>(experts, counts, hist, n, per, k, E, tile, cap, slot, src, seg,
                                                                           tile_expert, num_mtiles);
  }
  return static_cast<int>(cudaGetLastError());
}
extern "C" int vb_moe_plan(const void* experts, int wide, const int* counts, int* hist, int n, int k, int E, int tile, int cap, int* slot,
                           int* src, int* seg, int* tile_expert, int* num_mtiles, cudaStream_t s) {
  if (n <= 0 || k <= 0 || E <= 0 || E > 1024 || tile <= 0 || cap % tile) return -1;
  return wide ? moe_plan_launch(reinterpret_cast<const long long*>(experts), counts, hist, n, k, E, tile, cap, slot, src, seg, tile_expert, num_mtiles, s)
              : moe_plan_launch(reinterpret_cast<const int*>(experts), counts, hist, n, k, E, tile, cap, slot, src, seg, tile_expert, num_mtiles, s);
}

extern "C" int vb_moe_combine(const void* y, long long ldy, const int* slot, const float* w, void* out, long long ldo, int T, int H,
                              int k, cudaStream_t s) {
  if (T <= 0) return 0;
  if (H % 8 || ldy % 8 || ldo % 8) return -1;
  const long long n = static_cast<long long>(T) * (H / 8);
  moe_combine_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(y), ldy, slot, w,
                                                                       reinterpret_cast<__nv_bfloat16*>(out), ldo, T, H, k);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_combine_bwd_w(const void* g, long long ldg, const void* y, long long ldy, const int* slot, float* gw, int T,
                                    int H, int k, cudaStream_t s) {
  if (T <= 0) return 0;
  if (H % 8 || ldg % 8 || ldy % 8) return -1;
  const long long threads = static_cast<long long>(T) * k * 32;
  moe_combine_bwd_w_kernel<<<static_cast<int>((threads + 255) / 256), 256, 0, s>>>(
      reinterpret_cast<const __nv_bfloat16*>(g), ldg, reinterpret_cast<const __nv_bfloat16*>(y), ldy, slot, gw, T, H, k);
  return static_cast<int>(cudaGetLastError());
}
