// Causal GQA attention backward over packed (varlen) sequences on tcgen05 tensor cores (head_dim 64 and 128).
//
// One CTA = one (sequence, block of 128 keys, KV head, share of the GQA group's query heads). K and V of the block stay in shared memory
// and dK, dV stay in TMEM for the whole CTA, which walks over its query heads and every block of 64 queries at or
// below the diagonal. Everything is computed in the transposed frame so that the 128 keys are the M (TMEM lane)
// dimension and softmax threads own one key row each:
//
//   S^T  = K  Q^T            [128 keys, 64 q]   A = K  (K-major)     B = Q  (K-major)
//   dP^T = V  dO^T           [128 keys, 64 q]   A = V  (K-major)     B = dO (K-major)
//   P^T  = exp2(S^T * c - lse2[q]) (causal),   dS^T = P^T o (dP^T - D[q]) * scale          -> bf16, shared memory
//   dV  += P^T  dO           [128 keys, hd]     A = P^T  (K-major)   B = dO (MN-major)       TMEM-resident
//   dK  += dS^T Q            [128 keys, hd]     A = dS^T (K-major)   B = Q  (MN-major)       TMEM-resident
//   dQ^T = K^T dS^T          [hd, 64 q]         A = K  (MN-major)    B = dS^T (MN-major)     -> added to dQ in fp32
//
// dQ^T has two TMEM buffers: the additions of step i run after the softmax warps have handed P^T / dS^T of step i + 1 to
// the MMA warp, i.e. under the tensor-core work of step i + 1 instead of in front of it.
// Grid = (KV head, sequence, key block counted from the END of the sequence, longest first): blocks are handed out in
// order of decreasing work (the first key block meets every query block, the last one only its own), which keeps the
// tail of the launch short.
//
//   warp 0      TMA: K, V once; Q and dO tiles through a ring of 3 (head_dim 128) or 4 stages: under the load of all SMs a tile takes
//               longer than half a step to arrive; with two stages 5 x 3072 tokens, 28 / 4 heads, took 1723 us, now 1614
//   warp 1      MMA issue (one elected thread)
//   warps 2..9  two threads per key row (32 of the step's 64 queries each): tcgen05.ld S^T / dP^T -> P^T, dS^T ->
//               swizzled shared memory; drain dQ^T: a warp's 32 queries x 32 head-dim elements transposed through shared memory
//               into one TMA reduction (32 red.add per thread and step in place of it: 1862 us for 5 x 3072 tokens, now
//               1723); final dV (warps 2..5) / dK (warps 6..9) store
// D[q] = sum_d dO[q,d] O[q,d] comes from a small pre-pass; dQ, dK and dV leave in fp32 and a last pass turns them into the bf16 gradient
// of the projection output, undoing the rotary embedding on the way (attn_bwd_finish_kernel).
//
// Head_dim 64: dQ^T has 64 rows, but the tensor core's M stays 128 (with M = 64 the rows would sit on half of the lanes of every warp):
// A's second panel of 64 rows is the V tile, which lies right behind K in shared memory with the stride of a K panel, and the lanes
// 64..127 of the result are never read. 4 of 24 MMAs of a step are spent on them.
//
// A step takes microseconds and the first key block of a sequence meets every query block of every head of its group, so that a launch
// could not end before that one CTA: 14 heads of 64 over 2 KV heads, 12 sequences of about 1,000 tokens, had 192 CTAs of up to 160 steps
// where the average SM has 82 to do. The group's heads are therefore dealt to several CTAs (hsplit, see vb_attn_bwd) which add their
// dK / dV in fp32: 16-byte reductions, four neighbouring elements of a key row. Whole backward, before all three changes and now:
// that case 470 -> 295 us, two prompts with five continuations each (7,900 tokens, 28 / 4 heads of 128) 984 -> 800, 5 x 3072 1862 -> 1614,
// 8192 2491 -> 1983 us. A step of 64 queries still takes 2.5 us of which the tensor pipe works 1.1: S^T / dP^T of the next step, the
// softmax and the products of this one follow each other, and TMEM (512 columns at head_dim 128) has no room for a second S^T / dP^T.
// dQ, and dK / dV where several CTAs add to them, are summed in an order that varies from run to run; full determinism takes the autograd form.
//
// With `parent` (see attention_fwd_tcgen05.cu) a key block of a prompt has queries in several sequences. They are dealt to one CTA per
// (key block, query sequence): blockIdx.y = s is sequence s against its own keys, num_seqs + s is sequence s against those of parent[s],
// unmasked. dK / dV of a prompt, and only of a prompt, are then summed with fp32 atomics. One CTA per key block for all members would
// need no atomics but leave the launch waiting for the few prompt blocks: 434 steps against 174 on average for two groups of five.
#include "tcgen05_common.cuh"

#include <math.h>

namespace vb {

constexpr int AB_BK = 128;  // keys per CTA
constexpr int AB_BQ = 64;   // queries per step
constexpr int AB_THREADS = 320;  // TMA warp, MMA warp, eight softmax warps

struct AttnBwdParams {
  const int* cu_seqlens;
  const int* parent;   // [num_seqs] or null
  int num_seqs, nh, nkv, total_tokens, max_tiles;  // max_tiles: key blocks of the longest sequence
  int hsplit, heads_per;  // CTAs that share a group's query heads, heads of each
  const float* lse;    // [nh, T] natural log
  const float* delta;  // [nh, T]
  float* dq32;         // [T, nh*hd] fp32, zero on entry
  float* dk32;         // [T, nkv*hd] fp32; zero on entry with `parent` or hsplit > 1
  float* dv32;
  float scale, scale_log2;
  int* status;
};

template <int HD>
struct AttnBwdSmem {
  static constexpr int STAGES = HD == 128 ? 3 : 4;
  static constexpr int KV_BYTES = AB_BK * HD * 2;   // 32 KB each
  static constexpr int QO_BYTES = AB_BQ * HD * 2;   // 16 KB each, per stage
  static constexpr int PS_BYTES = AB_BK * AB_BQ * 2;  // 16 KB each
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + KV_BYTES;
  static constexpr int OFF_Q = OFF_V + KV_BYTES;
  static constexpr int OFF_DO = OFF_Q + STAGES * QO_BYTES;
  static constexpr int OFF_P = OFF_DO + STAGES * QO_BYTES;
  static constexpr int OFF_DS = OFF_P + PS_BYTES;
  static constexpr int OFF_VEC = OFF_DS + PS_BYTES;       // per softmax warp (8): [lse2 | delta][32] fp32
  static constexpr int OFF_DQ = OFF_VEC + 8 * 2 * 32 * 4;  // per softmax warp: 32 queries x 32 head-dim elements, fp32
  static constexpr int DQ_PIECE = 32 * 32 * 4;
  static constexpr int OFF_BAR = OFF_DQ + 8 * DQ_PIECE;
  // no alignment slack and no static shared memory: the dynamic window then starts 1024-byte aligned, which the kernel verifies
  static constexpr int TOTAL = OFF_BAR + 128;
  static_assert(TOTAL <= 232448, "shared memory of a CTA");
};

template <int HD>
__global__ void __launch_bounds__(AB_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_dq, const AttnBwdParams p) {
  using L = AttnBwdSmem<HD>;
  constexpr int PANELS = HD / 64;
  constexpr int STAGES = L::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem) & 1023u) != 0u) {  // the swizzled TMA / MMA layouts need 1024-byte aligned tiles
    if (threadIdx.x == 0) atomicExch(p.status, 9);
    return;
  }
  uint8_t* sK = smem + L::OFF_K;
  uint8_t* sV = smem + L::OFF_V;
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sDO = smem + L::OFF_DO;
  uint8_t* sP = smem + L::OFF_P;
  uint8_t* sDS = smem + L::OFF_DS;
  float* sVec = reinterpret_cast<float*>(smem + L::OFF_VEC);  // [8 warps][lse2 | delta][32]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* kv_full = bars;        // 1
  uint64_t* bar_sdp = bars + 1;    // S^T, dP^T ready
  uint64_t* bar_pds = bars + 2;    // P^T, dS^T written (8 warps)
  uint64_t* bar_dq = bars + 3;     // dV, dK, dQ^T MMAs of a step done
  uint64_t* qdo_full = bars + 4;   // [STAGES]
  uint64_t* qdo_empty = bars + 8;  // [STAGES]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 12);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = static_cast<int>(blockIdx.x) / p.hsplit, part = static_cast<int>(blockIdx.x) - kvh * p.hsplit;
  const int G = p.nh / p.nkv;
  const int head0 = kvh * G + part * p.heads_per, heads = min(p.heads_per, G - part * p.heads_per);  // at least one: see the launcher
  // query sequence, and the sequence of its keys: itself, or its parent
  const bool cross = static_cast<int>(blockIdx.y) >= p.num_seqs;
  const int qs = static_cast<int>(blockIdx.y) - (cross ? p.num_seqs : 0);
  const int ks = cross ? p.parent[qs] : qs;
  if (ks < 0 || ks >= p.num_seqs) return;  // no parent: uniform over the CTA, nothing allocated yet
  const int seq_start = p.cu_seqlens[qs], seqlen = p.cu_seqlens[qs + 1] - seq_start;
  const int key_start = p.cu_seqlens[ks], keylen = p.cu_seqlens[ks + 1] - key_start;
  const int from_end = p.max_tiles - 1 - static_cast<int>(blockIdx.z);
  const int ntiles = (keylen + AB_BK - 1) / AB_BK;
  if (ntiles > p.max_tiles && blockIdx.z == 0 && threadIdx.x == 0) atomicExch(p.status, ST_BAD_ARGS);  // max_seqlen too small
  if (from_end >= ntiles || seqlen <= 0) return;  // shorter sequence
  bool has_child = false;  // of the sequences that this thread looks at
  if (p.parent != nullptr && !cross)
    for (int s = threadIdx.x; s < p.num_seqs; s += AB_THREADS) has_child |= p.parent[s] == ks;
  const int k0 = (ntiles - 1 - from_end) * AB_BK;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_do);
    mbar_init(kv_full, 1);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&qdo_full[i], 1);
      mbar_init(&qdo_empty[i], 1);
    }
    mbar_init(bar_sdp, 1);
    mbar_init(bar_pds, 8);
    mbar_init(bar_dq, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  // dK / dV of this block are also written by CTAs of other heads, or of sequences that continue this one, wherever they stand
  const bool shared_keys = (__syncthreads_or(has_child) != 0) || p.hsplit > 1 || cross;
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const int i0 = cross ? 0 : k0 / AB_BQ;                        // first query block at or below the diagonal
  const int nqb = (seqlen + AB_BQ - 1) / AB_BQ;
  const int per_head = nqb - i0;
  const int n_it = per_head * heads;
  constexpr uint32_t TM_DV = 0, TM_DK = HD, TM_S = 2 * HD, TM_DP = 2 * HD + AB_BQ, TM_DQ = 2 * HD + 2 * AB_BQ;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * L::KV_BYTES);
#pragma unroll
      for (int c = 0; c < PANELS; ++c) {
        tma_load_2d(sK + c * (AB_BK * 128), &tm_k, kv_full, kvh * HD + 64 * c, key_start + k0);
        tma_load_2d(sV + c * (AB_BK * 128), &tm_v, kv_full, kvh * HD + 64 * c, key_start + k0);
      }
      for (int it = 0; it < n_it; ++it) {
        const int st = it % STAGES;
        if (!mbar_wait(&qdo_empty[st], ((it / STAGES) & 1) ^ 1)) {
          atomicExch(p.status, ST_TIMEOUT_PRODUCER);
          break;
        }
        const int head = head0 + it / per_head;
        const int q0 = (i0 + it % per_head) * AB_BQ;
        mbar_expect_tx(&qdo_full[st], 2 * L::QO_BYTES);
#pragma unroll
        for (int c = 0; c < PANELS; ++c) {
          tma_load_2d(sQ + st * L::QO_BYTES + c * (AB_BQ * 128), &tm_q, &qdo_full[st], head * HD + 64 * c, seq_start + q0);
          tma_load_2d(sDO + st * L::QO_BYTES + c * (AB_BQ * 128), &tm_do, &qdo_full[st], head * HD + 64 * c, seq_start + q0);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0 && n_it > 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(AB_BK, AB_BQ, false, false);   // S^T, dP^T
      constexpr uint32_t idesc_kv = make_idesc_f16(AB_BK, HD, false, true);      // dV, dK
      constexpr uint32_t idesc_dq = make_idesc_f16(128, AB_BQ, true, true);      // dQ^T (M = hd, padded to 128)
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aP = smem_u32(sP), aDS = smem_u32(sDS);
      auto issue_sdp = [&](int it) {
        const int st = it % STAGES;
        if (!mbar_wait(&qdo_full[st], (it / STAGES) & 1)) return false;
        tc_fence_after();
        const uint32_t bQ = smem_u32(sQ + st * L::QO_BYTES), bDO = smem_u32(sDO + st * L::QO_BYTES);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint64_t da = make_smem_desc_sw128(aK + (k >> 2) * (AB_BK * 128) + (k & 3) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(bQ + (k >> 2) * (AB_BQ * 128) + (k & 3) * 32, 16, 1024);
          tc_mma_f16_ss(tmem_base + TM_S, da, db, idesc_s, k > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint64_t da = make_smem_desc_sw128(aV + (k >> 2) * (AB_BK * 128) + (k & 3) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(bDO + (k >> 2) * (AB_BQ * 128) + (k & 3) * 32, 16, 1024);
          tc_mma_f16_ss(tmem_base + TM_DP, da, db, idesc_s, k > 0 ? 1u : 0u);
        }
        tc_commit(bar_sdp);
        return true;
      };
      bool ok = mbar_wait(kv_full, 0);
      if (ok) ok = issue_sdp(0);
      for (int it = 0; it < n_it && ok; ++it) {
        if (!mbar_wait(bar_pds, it & 1)) { ok = false; break; }
        tc_fence_after();
        if (it + 1 < n_it) ok = issue_sdp(it + 1);  // S^T/dP^T columns are free: the softmax of `it` has read them
        if (!ok) break;
        const int st = it % STAGES;
        const uint32_t bQ = smem_u32(sQ + st * L::QO_BYTES), bDO = smem_u32(sDO + st * L::QO_BYTES);
#pragma unroll
        for (int k = 0; k < AB_BQ / 16; ++k) {  // contraction over the 64 queries of the step
          const uint64_t dp = make_smem_desc_sw128(aP + k * 32, 16, 1024);
          const uint64_t dds = make_smem_desc_sw128(aDS + k * 32, 16, 1024);
          const uint64_t bdo = make_smem_desc_sw128(bDO + k * 2048, AB_BQ * 128, 1024);
          const uint64_t bq = make_smem_desc_sw128(bQ + k * 2048, AB_BQ * 128, 1024);
          tc_mma_f16_ss(tmem_base + TM_DV, dp, bdo, idesc_kv, (it > 0 || k > 0) ? 1u : 0u);
          tc_mma_f16_ss(tmem_base + TM_DK, dds, bq, idesc_kv, (it > 0 || k > 0) ? 1u : 0u);
        }
#pragma unroll
        for (int k = 0; k < AB_BK / 16; ++k) {  // contraction over the 128 keys
          const uint64_t da = make_smem_desc_sw128(aK + k * 2048, AB_BK * 128, 1024);
          const uint64_t db = make_smem_desc_sw128(aDS + k * 2048, AB_BK * 128, 1024);
          tc_mma_f16_ss(tmem_base + TM_DQ + (it & 1) * AB_BQ, da, db, idesc_dq, k > 0 ? 1u : 0u);
        }
        tc_commit(&qdo_empty[st]);
        tc_commit(bar_dq);
      }
      if (!ok) atomicExch(p.status, ST_TIMEOUT_MMA);
    }
  } else if (n_it > 0) {
    // ------------------------------------------------------------------ softmax backward / drains
    // Eight warps: warp w serves TMEM lane quarter w % 4 (thread == key row) and the query columns of half (w - 2) / 4,
    // so every key row is shared by two threads that never need each other's values.
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;   // 0: query columns 0..31 of the step, 1: columns 32..63
    const int r = q * 32 + lane;
    const int key = k0 + r;  // key index inside the sequence; also the head-dim index when draining dQ^T
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    const int cbase = half * 32;
    bool ok = true;
    constexpr float LOG2E = 1.4426950408889634f;

    float* dq_piece = reinterpret_cast<float*>(smem + L::OFF_DQ + (warp - 2) * L::DQ_PIECE);
    auto drain_dq = [&](int it) {
      if (HD < 128 && q * 32 >= HD) return;  // lanes of the padding rows
      const int head = head0 + it / per_head;
      const int q0 = (i0 + it % per_head) * AB_BQ + cbase;
      uint32_t v[32];
      tmem_ld_32x32(tmem_base + TM_DQ + (it & 1) * AB_BQ + cbase + lane_off, v);
      tmem_ld_wait();
      if (q0 >= seqlen) return;
      if (q0 + 32 > seqlen) {  // the rows behind belong to another sequence
        const long long row_stride = static_cast<long long>(p.nh) * HD;
        float* base = p.dq32 + static_cast<long long>(seq_start + q0) * row_stride + static_cast<long long>(head) * HD + r;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (q0 + j < seqlen) atomicAdd(base + j * row_stride, __uint_as_float(v[j]));
        }
        return;
      }
      if (lane == 0) tma_store_wait_read<0>();  // the reduction of the step before has read the piece
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 32; ++j) dq_piece[j * 32 + lane] = __uint_as_float(v[j]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_reduce_add_2d(&tm_dq, dq_piece, head * HD + q * 32, seq_start + q0);
        tma_store_commit();
      }
    };

    // lse (log2 domain) and delta of this warp's 32 queries of a step, one query per lane; fetched one step ahead
    float nl2 = 0.f, nde = 0.f;
    auto fetch_vec = [&](int it) {
      const int qi = (i0 + it % per_head) * AB_BQ + cbase + lane;
      nl2 = 0.f;
      nde = 0.f;
      if (it < n_it && qi < seqlen) {
        const long long o = static_cast<long long>(head0 + it / per_head) * p.total_tokens + seq_start + qi;
        nl2 = p.lse[o] * LOG2E;
        nde = p.delta[o] * p.scale;
      }
    };
    fetch_vec(0);
    for (int it = 0; it < n_it && ok; ++it) {
      const int q0 = (i0 + it % per_head) * AB_BQ;
      // a private copy per warp, so no barrier across warps is needed (a warp that gave up on a wait cannot leave the
      // others stuck)
      float* vL = sVec + (warp - 2) * 64;
      float* vD = vL + 32;
      __syncwarp();  // the step before has been read
      vL[lane] = nl2;
      vD[lane] = nde;
      __syncwarp();
      fetch_vec(it + 1);
      if (!mbar_wait(bar_sdp, it & 1)) { ok = false; break; }
      tc_fence_after();
      uint32_t pk[16], dk[16];  // packed bf16 pairs of P^T and dS^T: this key row, this warp's 32 queries
      {
        uint32_t s[32], dp[32];
        tmem_ld_32x32(tmem_base + TM_S + cbase + lane_off, s);
        tmem_ld_32x32(tmem_base + TM_DP + cbase + lane_off, dp);
        tmem_ld_wait();
        // only the blocks on the diagonal and the last (partial) query block of the sequence need the mask
        const bool masked = (!cross && q0 < k0 + AB_BK) || (q0 + AB_BQ > seqlen) || (cross && k0 + AB_BK > keylen);
        const float4* vL4 = reinterpret_cast<const float4*>(vL);
        const float4* vD4 = reinterpret_cast<const float4*>(vD);
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const float4 l4 = vL4[c >> 2], d4 = vD4[c >> 2];
          const float lv[4] = {l4.x, l4.y, l4.z, l4.w}, dv_[4] = {d4.x, d4.y, d4.z, d4.w};
          float pv[4], dsv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float pe = exp2f(fmaf(__uint_as_float(s[c + u]), p.scale_log2, -lv[u]));
            if (masked) {
              const int qi = q0 + cbase + c + u;
              if (!((cross ? key < keylen : key <= qi) && (qi < seqlen))) pe = 0.f;
            }
            pv[u] = pe;
            dsv[u] = pe * fmaf(__uint_as_float(dp[c + u]), p.scale, -dv_[u]);  // delta is stored pre-multiplied by scale
          }
          pk[c >> 1] = pack_bf16x2(pv[0], pv[1]);
          pk[(c >> 1) + 1] = pack_bf16x2(pv[2], pv[3]);
          dk[c >> 1] = pack_bf16x2(dsv[0], dsv[1]);
          dk[(c >> 1) + 1] = pack_bf16x2(dsv[2], dsv[3]);
        }
      }
      tc_fence_before();
      if (it > 0) {
        // the P^T / dS^T buffers are still read by the MMAs of the previous step
        if (!mbar_wait(bar_dq, (it - 1) & 1)) { ok = false; break; }
        tc_fence_after();
      }
      uint8_t* prow = sP + r * 128;
      uint8_t* drow = sDS + r * 128;
#pragma unroll
      for (int c4 = 0; c4 < 4; ++c4) {  // this warp's four 16-byte chunks of the 128-byte row
        const int sw = ((half * 4 + c4) ^ (r & 7)) << 4;
        *reinterpret_cast<uint4*>(prow + sw) = make_uint4(pk[c4 * 4], pk[c4 * 4 + 1], pk[c4 * 4 + 2], pk[c4 * 4 + 3]);
        *reinterpret_cast<uint4*>(drow + sw) = make_uint4(dk[c4 * 4], dk[c4 * 4 + 1], dk[c4 * 4 + 2], dk[c4 * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_pds);
      if (it > 0) {
        // dQ^T of the previous step sits in the other TMEM buffer; its next writer is the MMA of step it + 1, which
        // waits for this warp's next arrival
        drain_dq(it - 1);
        tc_fence_before();
      }
    }
    if (ok) ok = mbar_wait(bar_dq, (n_it - 1) & 1);
    if (!ok) {
      if (lane == 0) atomicExch(p.status, ST_TIMEOUT_EPILOGUE);
    } else {
      tc_fence_after();
      drain_dq(n_it - 1);
      // dV (first four warps) and dK (last four) of this key block: exclusive to this CTA (plain stores) unless other sequences share
      // the keys; the TMEM loads are warp-wide, the stores are predicated on the key being inside the sequence
      const bool key_ok = key < keylen;
      const long long tok = static_cast<long long>(key_start) + key;
      float* dst = (half == 0 ? p.dv32 : p.dk32) + (tok * p.nkv + kvh) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_base + (half == 0 ? TM_DV : TM_DK) + c * 32 + lane_off, o);
        tmem_ld_wait();
        if (!key_ok) continue;
        if (shared_keys) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + c * 32 + i), "f"(__uint_as_float(o[i])),
                         "f"(__uint_as_float(o[i + 1])), "f"(__uint_as_float(o[i + 2])), "f"(__uint_as_float(o[i + 3])) : "memory");
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(dst + c * 32 + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        }
      }
    }
  }

  if (warp >= 2 && lane == 0) tma_store_wait_all<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; hd / 8 lanes per (token, head), 16 bytes each, so that a warp has 1 KB in flight
__global__ void __launch_bounds__(256)
attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ dout, long long lddo, const __nv_bfloat16* __restrict__ out, long long ldo,
                      float* __restrict__ delta, int T, int nh, int hd) {
  const int lanes = hd >> 3;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  const long long w = i / lanes;
  const int l = static_cast<int>(i - w * lanes);
  float s = 0.f;
  const bool ok = w < static_cast<long long>(T) * nh;
  const int t = static_cast<int>(w / nh), h = static_cast<int>(w % nh);
  if (ok) {
    const uint4 a = *reinterpret_cast<const uint4*>(dout + static_cast<long long>(t) * lddo + h * hd + l * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(out + static_cast<long long>(t) * ldo + h * hd + l * 8);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s = fmaf(__uint_as_float(av[j] << 16), __uint_as_float(bv[j] << 16), s);
      s = fmaf(__uint_as_float(av[j] & 0xffff0000u), __uint_as_float(bv[j] & 0xffff0000u), s);
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (ok && l == 0) delta[static_cast<long long>(h) * T + t] = s;
}

// bf16 gradients from the fp32 sums: heads 0 .. nh of dq32, then nkv heads of dk32, then of dv32. With cos_t the q and k heads are
// rotated back by their token's position before they are rounded. Four pairs (d, d + hd / 2) per thread. One pass where the
// projection output's gradient used to take seven (cast of dq, copies of dq, dk and dv, rotations of q and k in place).
__global__ void __launch_bounds__(256)
attn_bwd_finish_kernel(const float* __restrict__ dq32, const float* __restrict__ dk32, const float* __restrict__ dv32,
                       __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, long long lddq,
                       long long lddk, long long lddv, const int* __restrict__ pos, const float* __restrict__ cos_t,
                       const float* __restrict__ sin_t, int T, int nh, int nkv, int hd) {
  const int half = hd >> 1, per_head = half >> 2, heads = nh + 2 * nkv;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  const long long item = i / per_head;
  if (item >= static_cast<long long>(T) * heads) return;
  const int d = static_cast<int>(i - item * per_head) * 4;
  const long long t = item / heads;
  const int h = static_cast<int>(item - t * heads);
  const float* src;
  __nv_bfloat16* dst;
  if (h < nh) {
    src = dq32 + (t * nh + h) * hd;
    dst = dq + t * lddq + h * hd;
  } else if (h < nh + nkv) {
    src = dk32 + (t * nkv + h - nh) * hd;
    dst = dk + t * lddk + (h - nh) * hd;
  } else {
    src = dv32 + (t * nkv + h - nh - nkv) * hd;
    dst = dv + t * lddv + (h - nh - nkv) * hd;
  }
  float4 a = *reinterpret_cast<const float4*>(src + d), b = *reinterpret_cast<const float4*>(src + half + d);
  if (cos_t != nullptr && h < nh + nkv) {
    const long long o = static_cast<long long>(pos[t]) * half + d;
    const float4 c = *reinterpret_cast<const float4*>(cos_t + o), sn = *reinterpret_cast<const float4*>(sin_t + o);
    const float4 x = a, y = b;
    a = make_float4(x.x * c.x + y.x * sn.x, x.y * c.y + y.y * sn.y, x.z * c.z + y.z * sn.z, x.w * c.w + y.w * sn.w);
    b = make_float4(y.x * c.x - x.x * sn.x, y.y * c.y - x.y * sn.y, y.z * c.z - x.z * sn.z, y.w * c.w - x.w * sn.w);
  }
  *reinterpret_cast<uint2*>(dst + d) = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
  *reinterpret_cast<uint2*>(dst + half + d) = make_uint2(pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
}

__device__ int g_attn_bwd_status[4];

}  // namespace vb

using namespace vb;

namespace vb {
template <int HD>
static cudaError_t launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                   const CUtensorMap& tdq, const AttnBwdParams& p, cudaStream_t stream) {
  auto kern = attn_bwd_kernel<HD>;
  constexpr int smem = AttnBwdSmem<HD>::TOTAL;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const dim3 grid(p.nkv * p.hsplit, p.num_seqs * (p.parent != nullptr ? 2 : 1), p.max_tiles);
  kern<<<grid, AB_THREADS, smem, stream>>>(tq, tk, tv, tdo, tdq, p);
  return cudaGetLastError();
}
}  // namespace vb

// Workspaces (caller-provided, any content): delta [nh*T], dq32 [T*nh*hd], dkv32 [2*T*nkv*hd], all fp32.
// q/dout/out: [T, nh, hd] views, k/v: [T, nkv, hd] views; dq/dk/dv are written with their own row strides. With pos / cos_t / sin_t
// (tables [*, hd/2]) the gradients are those in front of the rotary embedding. max_seqlen: of the sequences as cu_seqlens cuts them.
extern "C" int vb_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, long long ldq,
                           long long ldk, long long ldv, long long ldo, long long lddo, const float* lse,
                           const int* cu_seqlens, const int* parent, int num_seqs, int total_tokens, int nh, int nkv, int hd, float scale,
                           void* dq, void* dk, void* dv, long long lddq, long long lddk, long long lddv, const int* pos,
                           const float* cos_t, const float* sin_t, float* delta_ws, float* dq32_ws, float* dkv32_ws, int max_seqlen,
                           cudaStream_t stream) {
  if (total_tokens <= 0 || num_seqs <= 0) return 0;
  if (max_seqlen <= 0 || num_seqs > (parent != nullptr ? 32767 : 65535)) return -4;
  if (hd != 64 && hd != 128) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (ldo % 8) || (lddo % 8) || (lddq % 8) || (lddk % 8) || (lddv % 8) || (nh % nkv)) return -1;
  CUtensorMap tq, tk, tv, tdo, tdq;
  const auto bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  if (!make_tmap_2d(&tq, q, bf, 2, total_tokens, (uint64_t)nh * hd, ldq, 64, AB_BQ, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  if (!make_tmap_2d(&tdo, dout, bf, 2, total_tokens, (uint64_t)nh * hd, lddo, 64, AB_BQ, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  if (!make_tmap_2d(&tk, k, bf, 2, total_tokens, (uint64_t)nkv * hd, ldk, 64, AB_BK, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  if (!make_tmap_2d(&tv, v, bf, 2, total_tokens, (uint64_t)nkv * hd, ldv, 64, AB_BK, CU_TENSOR_MAP_SWIZZLE_128B)) return -3;
  if (!make_tmap_2d(&tdq, dq32_ws, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, total_tokens, (uint64_t)nh * hd, (uint64_t)nh * hd, 32, 32,
                    CU_TENSOR_MAP_SWIZZLE_NONE)) return -3;
  static int* status = nullptr;
  if (status == nullptr) cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_attn_bwd_status);
  const long long T = total_tokens, lanes = T * nh * (hd / 8);
  attn_bwd_delta_kernel<<<static_cast<int>((lanes + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(dout), lddo, reinterpret_cast<const __nv_bfloat16*>(out), ldo, delta_ws,
      total_tokens, nh, hd);
  float* dk32 = dkv32_ws;
  float* dv32 = dkv32_ws + T * nkv * hd;
  cudaError_t e = cudaMemsetAsync(dq32_ws, 0, sizeof(float) * static_cast<size_t>(T) * nh * hd, stream);
  // Shares that a group's heads are dealt in: the number whose launch is estimated shortest. A CTA takes its steps and about three more
  // (set-up, loads of K and V, dK and dV out: with sequences of 40 tokens that is most of it). A launch takes as long as its longest CTA, the
  // first key block of the longest sequence, or as an SM's share of all CTAs and some of what comes last: a quarter of a last key block,
  // or, with parents, most of a long CTA, because queries behind a prompt meet its last key blocks as often as its first. Only the longest
  // sequence is known here, so total_tokens / max_seqlen sequences of that length stand for all, and a continuation for a CTA per key block.
  // Best share, its time and that of one share, 28 / 4 heads of 128: 64 x 40 tokens 1 (78 us; 104 with four), 8 x 1000 1 (393; 411 with two),
  // 5 x 1000 2 (267; 339), 3 x 1000 4 (168; 318), 1 x 3072 4 (327; 820), 1 x 200 7 (27; 90); two prompts with five continuations 2 (792; 825);
  // 32 / 8 heads, three prompts of 900 with eight continuations of 50 1 (411; 519 with two). Within 6% of the best share over 33 shapes, heads
  // of 64 among them.
  const int G = nh / nkv, sms = num_sms();
  const double qb = (max_seqlen + AB_BQ - 1) / AB_BQ, kb = (max_seqlen + AB_BK - 1) / AB_BK, extra = 3.0;
  const double seqs = total_tokens > max_seqlen ? static_cast<double>(total_tokens) / max_seqlen : 1.0;
  const double blocks = kb * (seqs + (parent != nullptr ? num_seqs : 0));
  int hsplit = 1;
  double shortest = 0.0;
  for (int share = 1; share <= G; ++share) {
    const int per = (G + share - 1) / share;
    if ((G + per - 1) / per != share) continue;  // deals the heads as fewer shares do
    const double longest = per * qb + extra;
    const double mean = nkv * (seqs * G * kb * (qb - kb + 1) + share * blocks * extra) / sms;
    const double all = mean + (parent != nullptr ? 0.75 * longest : 0.25 * (2 * per + extra));
    const double est = longest > all ? longest : all;
    if (share == 1 || est < shortest) {
      shortest = est;
      hsplit = share;
    }
  }
  const int heads_per = (G + hsplit - 1) / hsplit;
  if (e == cudaSuccess && (parent != nullptr || hsplit > 1)) e = cudaMemsetAsync(dkv32_ws, 0, sizeof(float) * 2 * static_cast<size_t>(T) * nkv * hd, stream);
  if (e != cudaSuccess) return static_cast<int>(e);
  AttnBwdParams p{};
  p.cu_seqlens = cu_seqlens; p.parent = parent; p.num_seqs = num_seqs; p.nh = nh; p.nkv = nkv; p.total_tokens = total_tokens;
  p.lse = lse; p.delta = delta_ws; p.dq32 = dq32_ws; p.dk32 = dk32; p.dv32 = dv32;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  p.max_tiles = (max_seqlen + AB_BK - 1) / AB_BK;
  p.hsplit = hsplit; p.heads_per = heads_per;
  if (p.max_tiles > 65535) return -4;
  e = hd == 128 ? launch_attn_bwd<128>(tq, tk, tv, tdo, tdq, p, stream) : launch_attn_bwd<64>(tq, tk, tv, tdo, tdq, p, stream);
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long n = T * (nh + 2 * nkv) * (hd / 8);
  attn_bwd_finish_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, stream>>>(
      dq32_ws, dk32, dv32, reinterpret_cast<__nv_bfloat16*>(dq), reinterpret_cast<__nv_bfloat16*>(dk), reinterpret_cast<__nv_bfloat16*>(dv),
      lddq, lddk, lddv, pos, cos_t, sin_t, total_tokens, nh, nkv, hd);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int vb_attn_bwd_status() {
  int h[4] = {0, 0, 0, 0};
  if (cudaMemcpyFromSymbol(h, g_attn_bwd_status, sizeof(h)) != cudaSuccess) return -1;
  if (h[0] != 0) {
    int z[4] = {0, 0, 0, 0};
    cudaMemcpyToSymbol(g_attn_bwd_status, z, sizeof(z));
  }
  return h[0];
}
