// GEMMs whose rows come in tiles of 16 to 128 tokens: fp8 (e4m3) with 1x128 block scaling on both operands, plain or grouped by expert,
// and the bf16 product of a mixture-of-experts layer with few tokens per expert. Also the quantisers that produce fp8 operands.
//
//   fp8:  D[m, n] (bf16) = sum over 128-wide K blocks kb of  sx[kb, m] * sw[kb, n] * ( Xq[m, kb] . Wq[n, kb] )
//   bf16: D[m, n] (bf16) = X[m, :] . W[n, :]
//
// Xq [M, K], Wq [N, K] are e4m3, K-major, K % 128 == 0. Scales are fp32 and stored block-major: sx [K/128, M], sw [K/128, N].
//
// The product is computed transposed: 128 weight rows are the M axis of the MMA, a tile of R = 16, 32, 64 or 128 tokens its N axis. A
// decode step of a mixture-of-experts layer (32 tokens, 8 of 128 experts each) has about two tokens per expert and is bound by reading
// the weights of ~110 experts once; tiles of 128 tokens made it pad, write, quantise and read 60 times the rows. A persistent grid
// walks over (token tile, weight tile) with one ring of 6 to 10 stages, so that the loads of the next tile run under the end of the
// last one. The scales of a stage travel with its operands (cp.async into the same stage, counted on the same barrier): fetched by the
// epilogue when it needed them they were a serial chain of one memory latency per K block.
// With many tokens: 8192 x 5120 x 2048 217 us (397 with 128 x 128 tiles, a scale fetch per block and rows stored by their thread), 2000 x 37888 x
// 3584 597 us (2086).
// A decode step of Qwen3-30B-A3B, 32 tokens, fp8: the two products of a layer's experts (523 MB of weights) 103 us (5.1 TB/s); they and
// the two dense projections together 790 -> 130 us.
//
//   warp 0      producer: TMA of a weight tile (128 rows x 128 bytes) and a token tile (R x 128 bytes), cp.async of their scales
//   warp 1      MMA issue; fp8: into one of two TMEM buffers per K block (the block's scale factors differ per row and column);
//               bf16: one of two buffers per output tile
//   warps 2..   epilogue, thread == weight row (R >= 32: two threads, half of the tokens each): tcgen05.ld, fp8: times sw[n] * sx[m] into
//               fp32 registers; after the last block store column by column (64 bytes of a token's row per warp)
#include "tcgen05_common.cuh"

#include <cuda_fp8.h>
#include <math.h>

namespace vb {

constexpr int TG_BM = 128;   // weight rows per tile
constexpr int TG_BK = 128;   // bytes of K per stage

struct TileGemmParams {
  int M, N, K;                  // tokens (rows of X), output columns, depth in elements
  int ntiles;                   // weight tiles of one matrix
  int mtiles;                   // token tiles (grouped: upper bound)
  const float* sx;              // [K/128, M]
  const float* sw;              // [K/128, ldsw]
  long long ldsw;               // N, or E * N when grouped
  __nv_bfloat16* D;
  long long ldd;
  const __nv_bfloat16* bias;
  int* status;
  const int* tile_expert;       // grouped: expert of token tile i; W holds E stacked [N, K] matrices. nullptr = plain
  const int* num_mtiles;        // grouped: device scalar, tiles in use
};

template <bool FP8, int R>
struct TileGemm {
  static constexpr int STAGES = R <= 32 ? 10 : (R == 64 ? 8 : 6);
  static constexpr int W_BYTES = TG_BM * TG_BK, X_BYTES = R * TG_BK;
  static constexpr int SC_BYTES = FP8 ? 1024 : 0;  // 128 weight scales, then R token scales
  static constexpr int STAGE = W_BYTES + X_BYTES + SC_BYTES;
  static constexpr int EW = R >= 32 ? 8 : 4;       // epilogue warps
  static constexpr int COLS = R / (EW / 4);        // tokens per epilogue thread
  static constexpr int THREADS = 64 + 32 * EW;
  static constexpr int TMEM_COLS = 2 * R < 32 ? 32 : 2 * R;
  static constexpr int OFF_BAR = STAGES * STAGE;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
  static_assert(TOTAL <= 232448, "shared memory of a CTA");
};

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// arrives on `bar` (counted in its init) once the thread's cp.async so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <bool FP8, int R>
__global__ void __launch_bounds__(TileGemm<FP8, R>::THREADS, 1)
tile_gemm_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w, const TileGemmParams p) {
  using L = TileGemm<FP8, R>;
  constexpr int STAGES = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* full_bar = bars;                    // [STAGES]
  uint64_t* empty_bar = bars + STAGES;          // [STAGES]
  uint64_t* acc_full = bars + 2 * STAGES;       // [2]
  uint64_t* acc_empty = bars + 2 * STAGES + 2;  // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = FP8 ? p.K / 128 : (p.K + 63) / 64;
  const int mtiles = p.tile_expert != nullptr ? min(*p.num_mtiles, p.mtiles) : p.mtiles;
  const int items = mtiles * p.ntiles;
  if (static_cast<int>(blockIdx.x) >= items) return;  // uniform over the CTA; nothing allocated yet

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_x);
    tma_prefetch_desc(&tma_w);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], FP8 ? 1 + 32 : 1);           // the TMA's expectation, and every lane's scales
      mbar_init(&empty_bar[s], FP8 ? 1 + L::EW : 1);       // the MMAs, and the readers of the scales
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], L::EW);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (all lanes: they carry the scales)
    int st = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
      const int mt = it / p.ntiles, n0 = (it - mt * p.ntiles) * TG_BM;
      const int w_row0 = (p.tile_expert != nullptr ? p.tile_expert[mt] * p.N : 0) + n0;
      const int m0 = mt * R;
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[st], phase ^ 1));
        if (!ok) break;
        uint8_t* sw = smem + st * L::STAGE;
        if (lane == 0) {
          mbar_expect_tx(&full_bar[st], L::W_BYTES + L::X_BYTES);
          const int k0 = kb * (FP8 ? 128 : 64);
          tma_load_2d(sw, &tma_w, &full_bar[st], k0, w_row0);
          tma_load_2d(sw + L::W_BYTES, &tma_x, &full_bar[st], k0, m0);
        }
        if constexpr (FP8) {
          float* sc = reinterpret_cast<float*>(sw + L::W_BYTES + L::X_BYTES);
          // N % 8 == 0: the 16-byte pieces are aligned and inside or outside as a whole
          if (n0 + lane * 4 < p.N) cp_async16(sc + lane * 4, p.sw + static_cast<long long>(kb) * p.ldsw + w_row0 + lane * 4);
#pragma unroll
          for (int u = 0; u < (R + 31) / 32; ++u) {
            const int j = u * 32 + lane;
            if (j < R && m0 + j < p.M) cp_async4(sc + TG_BM + j, p.sx + static_cast<long long>(kb) * p.M + m0 + j);
          }
          cp_async_arrive(&full_bar[st]);
        }
        if (++st == STAGES) { st = 0; phase ^= 1; }
      }
    }
    if (!ok && lane == 0) atomicExch(p.status, ST_TIMEOUT_PRODUCER);
    if constexpr (FP8) asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = FP8 ? make_idesc_e4m3(TG_BM, R) : make_idesc_f16(TG_BM, R, false, false);
      int st = 0, buf = 0;
      uint32_t phase = 0, buf_phase = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb) {
          if ((FP8 || kb == 0) && !mbar_wait(&acc_empty[buf], buf_phase ^ 1)) { ok = false; break; }
          if (!mbar_wait(&full_bar[st], phase)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + st * L::STAGE), sx = sw + L::W_BYTES;
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // 32 bytes of K per instruction
            const uint64_t da = make_smem_desc_sw128(sw + k * 32, 16, 1024);
            const uint64_t db = make_smem_desc_sw128(sx + k * 32, 16, 1024);
            if constexpr (FP8) tc_mma_f8_ss(tmem_base + buf * R, da, db, idesc, k > 0 ? 1u : 0u);
            else tc_mma_f16_ss(tmem_base + buf * R, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          tc_commit(&empty_bar[st]);
          if (FP8 || kb == num_kb - 1) {
            tc_commit(&acc_full[buf]);
            if (++buf == 2) { buf = 0; buf_phase ^= 1; }
          }
          if (++st == STAGES) { st = 0; phase ^= 1; }
        }
      }
      if (!ok) atomicExch(p.status, ST_TIMEOUT_MMA);
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3, half = (warp - 2) >> 2;  // TMEM lane quarter, half of the tokens
    const int c0 = half * L::COLS;
    constexpr int CH = L::COLS < 32 ? 16 : 32;       // columns per tcgen05.ld
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    int st = 0, buf = 0;
    uint32_t phase = 0, buf_phase = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
      const int mt = it / p.ntiles, n = (it - mt * p.ntiles) * TG_BM + q * 32 + lane;
      float acc[L::COLS];
#pragma unroll
      for (int j = 0; j < L::COLS; ++j) acc[j] = 0.f;
      const int reps = FP8 ? num_kb : 1;
      for (int kb = 0; kb < reps; ++kb) {
        if (FP8 && !mbar_wait(&full_bar[st], phase)) { ok = false; break; }  // the stage's scales; passes once the MMAs have run
        if (!mbar_wait(&acc_full[buf], buf_phase)) { ok = false; break; }
        tc_fence_after();
        const float* sc = reinterpret_cast<const float*>(smem + st * L::STAGE + L::W_BYTES + L::X_BYTES);
        const float rw = FP8 ? sc[q * 32 + lane] : 1.f;
#pragma unroll
        for (int c = 0; c < L::COLS; c += CH) {
          uint32_t r[CH];
          if constexpr (CH == 16) tmem_ld_32x16(tmem_base + buf * R + c0 + c + lane_off, r);
          else tmem_ld_32x32(tmem_base + buf * R + c0 + c + lane_off, r);
          tmem_ld_wait();
          if constexpr (FP8) {
            const float4* sx4 = reinterpret_cast<const float4*>(sc + TG_BM + c0 + c);
#pragma unroll
            for (int j = 0; j < CH; j += 4) {
              const float4 s4 = sx4[j >> 2];
              acc[c + j] = fmaf(__uint_as_float(r[j]), rw * s4.x, acc[c + j]);
              acc[c + j + 1] = fmaf(__uint_as_float(r[j + 1]), rw * s4.y, acc[c + j + 1]);
              acc[c + j + 2] = fmaf(__uint_as_float(r[j + 2]), rw * s4.z, acc[c + j + 2]);
              acc[c + j + 3] = fmaf(__uint_as_float(r[j + 3]), rw * s4.w, acc[c + j + 3]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < CH; ++j) acc[c + j] = __uint_as_float(r[j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&acc_empty[buf]);
          if (FP8) mbar_arrive(&empty_bar[st]);
        }
        if (++buf == 2) { buf = 0; buf_phase ^= 1; }
        if (FP8 && ++st == STAGES) { st = 0; phase ^= 1; }
      }
      if (ok && n < p.N) {
        const float b = p.bias != nullptr ? __bfloat162float(p.bias[n]) : 0.f;
        const int m0 = mt * R + c0;
        __nv_bfloat16* d = p.D + static_cast<long long>(m0) * p.ldd + n;
#pragma unroll
        for (int j = 0; j < L::COLS; ++j)
          if (m0 + j < p.M) d[static_cast<long long>(j) * p.ldd] = __float2bfloat16(acc[j] + b);
      }
    }
    if (!ok && lane == 0) atomicExch(p.status, ST_TIMEOUT_EPILOGUE);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

template <bool FP8, int R>
static int launch_tile_gemm(const CUtensorMap& tx, const CUtensorMap& tw, const TileGemmParams& p, cudaStream_t stream) {
  using L = TileGemm<FP8, R>;
  auto kern = tile_gemm_kernel<FP8, R>;
  // on every launch: the attribute belongs to the current device, and a process may use several
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long items = static_cast<long long>(p.mtiles) * p.ntiles;
  const int sms = num_sms();
  kern<<<static_cast<int>(items < sms ? items : sms), L::THREADS, L::TOTAL, stream>>>(tx, tw, p);
  return static_cast<int>(cudaGetLastError());
}

// x [R, C] bf16 -> q [R, C] e4m3 and scales [C/128, R] fp32 with  x ~= q * scale,  scale = amax(block) / 448.
// One warp per (row, 128-column block): 4 elements per lane.
__global__ void fp8_quant_1x128_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ q, long long ldq,
                                       float* __restrict__ scales, int R, int C) {
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int nblk = C / 128;
  if (w >= static_cast<long long>(R) * nblk) return;
  const int r = static_cast<int>(w / nblk), b = static_cast<int>(w % nblk);
  const __nv_bfloat16* src = x + static_cast<long long>(r) * ldx + b * 128 + lane * 4;
  const uint2 raw = *reinterpret_cast<const uint2*>(src);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
  const float2 a = __bfloat1622float2(h[0]), c = __bfloat1622float2(h[1]);
  float amax = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(c.x), fabsf(c.y)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = fmaxf(amax, 1e-12f) / 448.f;
  const float inv = 1.f / scale;
  __nv_fp8x4_e4m3 packed(make_float4(a.x * inv, a.y * inv, c.x * inv, c.y * inv));
  *reinterpret_cast<uint32_t*>(q + static_cast<long long>(r) * ldq + b * 128 + lane * 4) = *reinterpret_cast<uint32_t*>(&packed);
  if (lane == 0) scales[static_cast<long long>(b) * R + r] = scale;
}

// The same quantisation fused with what produces its input, for the rows of the tiles in use (num_mtiles * tile_rows; null: all).
// One warp per (row, 128-column block).
__device__ __forceinline__ void quant_block(const float (&f)[4], uint8_t* q, float* scale, int lane) {
  float amax = fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fmaxf(fabsf(f[2]), fabsf(f[3])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float sc = fmaxf(amax, 1e-12f) / 448.f;
  const float inv = 1.f / sc;
  __nv_fp8x4_e4m3 packed(make_float4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv));
  *reinterpret_cast<uint32_t*>(q + lane * 4) = *reinterpret_cast<uint32_t*>(&packed);
  if (lane == 0) *scale = sc;
}

// q[r] = quantised src[map[r]], zeros where map[r] < 0
__global__ void __launch_bounds__(256)
moe_gather_quant_kernel(const __nv_bfloat16* __restrict__ src, long long lds, const int* __restrict__ map, uint8_t* __restrict__ q,
                        float* __restrict__ scales, int R, int C, const int* __restrict__ num_mtiles, int tile_rows) {
  const long long w = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, nblk = C / 128;
  const int r = static_cast<int>(w / nblk), b = static_cast<int>(w - static_cast<long long>(r) * nblk);
  if (r >= min(R, *num_mtiles * tile_rows)) return;
  const int s = map[r];
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  if (s >= 0) {
    const uint2 raw = *reinterpret_cast<const uint2*>(src + static_cast<long long>(s) * lds + b * 128 + lane * 4);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 x = __bfloat1622float2(h[0]), y = __bfloat1622float2(h[1]);
    f[0] = x.x; f[1] = x.y; f[2] = y.x; f[3] = y.y;
  }
  quant_block(f, q + static_cast<long long>(r) * C + b * 128, scales + static_cast<long long>(b) * R + r, lane);
}

// q = quantised silu(gate) * up of gu [R, 2 C] (rounded to bf16 in between, as the two kernels it replaces did)
__global__ void __launch_bounds__(256)
moe_swiglu_quant_kernel(const __nv_bfloat16* __restrict__ gu, uint8_t* __restrict__ q, float* __restrict__ scales, int R, int C,
                        const int* __restrict__ num_mtiles, int tile_rows) {
  const long long w = (blockIdx.x * 256LL + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, nblk = C / 128;
  const int r = static_cast<int>(w / nblk), b = static_cast<int>(w - static_cast<long long>(r) * nblk);
  if (r >= min(R, *num_mtiles * tile_rows)) return;
  const __nv_bfloat16* row = gu + static_cast<long long>(r) * 2 * C + b * 128 + lane * 4;
  const uint2 rg = *reinterpret_cast<const uint2*>(row), ru = *reinterpret_cast<const uint2*>(row + C);
  const __nv_bfloat162 *hg = reinterpret_cast<const __nv_bfloat162*>(&rg), *hu = reinterpret_cast<const __nv_bfloat162*>(&ru);
  const float2 g0 = __bfloat1622float2(hg[0]), g1 = __bfloat1622float2(hg[1]), u0 = __bfloat1622float2(hu[0]), u1 = __bfloat1622float2(hu[1]);
  const float g[4] = {g0.x, g0.y, g1.x, g1.y}, u[4] = {u0.x, u0.y, u1.x, u1.y};
  float f[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = __bfloat162float(__float2bfloat16(g[j] / (1.f + __expf(-g[j])) * u[j]));
  quant_block(f, q + static_cast<long long>(r) * C + b * 128, scales + static_cast<long long>(b) * R + r, lane);
}

// w [R, C] bf16 -> q [R, C] e4m3 and scale_inv [ceil(R/128), ceil(C/128)] fp32: one scale per 128 x 128 block
// (w ~= q * scale_inv, scale_inv = amax(block) / 448), the weight format of block-scaled fp8 checkpoints.
// One CTA of 256 threads per block: pass 1 reduces |w| over the block, pass 2 converts.
__global__ void fp8_quant_128x128_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, uint8_t* __restrict__ q, long long ldq,
                                         float* __restrict__ scale_inv, int R, int C) {
  __shared__ float s_red[8];
  __shared__ float s_scale;
  const int bc = blockIdx.x, br = blockIdx.y;
  const int r0 = br * 128, c0 = bc * 128;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // thread t covers columns (t % 32) * 4 .. +3 of rows (t / 32) + 8 * i
  const int col = c0 + (tid & 31) * 4;
  float amax = 0.f;
  float4 vals[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = r0 + (tid >> 5) + 8 * i;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < R && col < C) {  // C % 4 == 0: a 4-vector is inside or outside as a whole
      const uint2 raw = *reinterpret_cast<const uint2*>(w + static_cast<long long>(row) * ldw + col);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
      const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
      v = make_float4(a.x, a.y, b.x, b.y);
    }
    vals[i] = v;
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) s_red[warp] = amax;
  __syncthreads();
  if (tid == 0) {
    float m = s_red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) m = fmaxf(m, s_red[i]);
    const float sc = fmaxf(m, 1e-12f) / 448.f;
    s_scale = sc;
    scale_inv[static_cast<long long>(br) * gridDim.x + bc] = sc;
  }
  __syncthreads();
  const float inv = 1.f / s_scale;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = r0 + (tid >> 5) + 8 * i;
    if (row < R && col < C) {
      const float4 v = vals[i];
      __nv_fp8x4_e4m3 packed(make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv));
      *reinterpret_cast<uint32_t*>(q + static_cast<long long>(row) * ldq + col) = *reinterpret_cast<uint32_t*>(&packed);
    }
  }
}

__device__ int g_fp8_status[4];

}  // namespace vb

using namespace vb;

extern "C" int vb_fp8_quant_1x128(const void* x, long long ldx, void* q, long long ldq, float* scales, int R, int C, cudaStream_t s) {
  if (R <= 0 || C <= 0) return 0;
  if ((C % 128) || (ldx % 4) || (ldq % 4)) return -1;
  const long long threads = static_cast<long long>(R) * (C / 128) * 32;
  fp8_quant_1x128_kernel<<<static_cast<int>((threads + 255) / 256), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), ldx,
                                                                                 reinterpret_cast<uint8_t*>(q), ldq, scales, R, C);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_moe_gather_quant(const void* src, long long lds, const int* map, void* q, float* scales, int R, int C,
                                   const int* num_mtiles, int tile_rows, cudaStream_t s) {
  if (R <= 0 || C <= 0) return 0;
  if ((C % 128) || (lds % 4) || (reinterpret_cast<uintptr_t>(src) & 7)) return -1;
  const long long blocks = (static_cast<long long>(R) * (C / 128) + 7) / 8;
  moe_gather_quant_kernel<<<static_cast<int>(blocks), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(src), lds, map,
                                                                   reinterpret_cast<uint8_t*>(q), scales, R, C, num_mtiles, tile_rows);
  return static_cast<int>(cudaGetLastError());
}
extern "C" int vb_moe_swiglu_quant(const void* gu, void* q, float* scales, int R, int C, const int* num_mtiles, int tile_rows, cudaStream_t s) {
  if (R <= 0 || C <= 0) return 0;
  if (C % 128) return -1;
  const long long blocks = (static_cast<long long>(R) * (C / 128) + 7) / 8;
  moe_swiglu_quant_kernel<<<static_cast<int>(blocks), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(gu), reinterpret_cast<uint8_t*>(q),
                                                                   scales, R, C, num_mtiles, tile_rows);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_fp8_quant_128x128(const void* w, long long ldw, void* q, long long ldq, float* scale_inv, int R, int C, cudaStream_t s) {
  if (R <= 0 || C <= 0) return 0;
  if ((C % 4) || (ldw % 4) || (ldq % 4)) return -1;
  dim3 grid((C + 127) / 128, (R + 127) / 128);
  fp8_quant_128x128_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(w), ldw, reinterpret_cast<uint8_t*>(q), ldq,
                                                scale_inv, R, C);
  return static_cast<int>(cudaGetLastError());
}

// X [M, K], W [N, K] (grouped: E stacked matrices, w_rows = E * N), rows of X in tiles of R tokens.
template <bool FP8>
static int tile_gemm(const void* X, const float* sx, const void* W, const float* sw, void* D, const void* bias, int M, int N, int K, int E,
                     long long ldx, long long ldw, long long ldd, int R, const int* tile_expert, const int* num_mtiles, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || E <= 0) return 0;
  constexpr int eb = FP8 ? 1 : 2;
  const bool grouped = tile_expert != nullptr;
  if ((K % (FP8 ? 128 : 8)) || (N % 8) || ((ldx * eb) % 16) || ((ldw * eb) % 16) || (grouped && (M % R))) return -1;
  if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(sw)) & 15) return -2;
  const long long mtiles = (M + R - 1) / R, ntiles = (N + TG_BM - 1) / TG_BM;
  if (mtiles * ntiles > 0x7fffffffLL - 65536 || static_cast<long long>(E) * N > 0x7fffffffLL) return -4;
  CUtensorMap tx, tw;
  const auto dt = FP8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  if (!make_tmap_2d(&tx, X, dt, eb, M, K, ldx, TG_BK / eb, R, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  if (!make_tmap_2d(&tw, W, dt, eb, static_cast<uint64_t>(E) * N, K, ldw, TG_BK / eb, TG_BM, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  static int* status = nullptr;
  if (status == nullptr) cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_fp8_status);
  TileGemmParams p{};
  p.M = M; p.N = N; p.K = K; p.ntiles = static_cast<int>(ntiles); p.mtiles = static_cast<int>(mtiles);
  p.sx = sx; p.sw = sw; p.ldsw = static_cast<long long>(E) * N;
  p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.status = status;
  p.tile_expert = tile_expert; p.num_mtiles = num_mtiles;
  switch (R) {
    case 16: return launch_tile_gemm<FP8, 16>(tx, tw, p, stream);
    case 32: return launch_tile_gemm<FP8, 32>(tx, tw, p, stream);
    case 64: return launch_tile_gemm<FP8, 64>(tx, tw, p, stream);
    case 128: return launch_tile_gemm<FP8, 128>(tx, tw, p, stream);
  }
  return -1;
}

// The smallest token tile that covers the rows in one: the weights are read once.
extern "C" int vb_gemm_fp8_blockscale(const void* Aq, const float* sa, const void* Bq, const float* sb, void* D, const void* bias, int M,
                                      int N, int K, long long lda, long long ldb, long long ldd, cudaStream_t stream) {
  const int R = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  return tile_gemm<true>(Aq, sa, Bq, sb, D, bias, M, N, K, 1, lda, ldb, ldd, R, nullptr, nullptr, stream);
}

// Grouped variants for mixture-of-experts layers: D[rows, N] = A[rows, K] * B_e^T for the expert e of each tile of tile_rows rows
// (16, 32, 64 or 128; rows_cap a multiple of it).
//  B [E * N, K]; fp8: scales sa [K/128, rows_cap], sb [K/128, E * N];
//  tile_expert[i] = expert of tile i, num_mtiles (device scalar) = tiles in use. Rows of unused tiles are not written.
extern "C" int vb_gemm_fp8_blockscale_grouped(const void* Aq, const float* sa, const void* Bq, const float* sb, void* D, int rows_cap,
                                              int N, int K, int E, long long lda, long long ldb, long long ldd, int tile_rows,
                                              const int* tile_expert, const int* num_mtiles, cudaStream_t stream) {
  return tile_gemm<true>(Aq, sa, Bq, sb, D, nullptr, rows_cap, N, K, E, lda, ldb, ldd, tile_rows, tile_expert, num_mtiles, stream);
}
extern "C" int vb_gemm_bf16_grouped_tiles(const void* A, const void* B, void* D, int rows_cap, int N, int K, int E, long long lda,
                                          long long ldb, long long ldd, int tile_rows, const int* tile_expert, const int* num_mtiles,
                                          cudaStream_t stream) {
  return tile_gemm<false>(A, nullptr, B, nullptr, D, nullptr, rows_cap, N, K, E, lda, ldb, ldd, tile_rows, tile_expert, num_mtiles, stream);
}

extern "C" int vb_fp8_status() {
  int h[4] = {0, 0, 0, 0};
  if (cudaMemcpyFromSymbol(h, g_fp8_status, sizeof(h)) != cudaSuccess) return -1;
  if (h[0] != 0) {
    int z[4] = {0, 0, 0, 0};
    cudaMemcpyToSymbol(g_fp8_status, z, sizeof(z));
  }
  return h[0];
}
