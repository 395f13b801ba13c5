// Single-pass flash-attention backward on CTA PAIRS (tcgen05.mma.cta_group::2): dQ, dK and dV of 256 keys per pair.
//
// What bounds the single-CTA kernel (attention_bwd_fused_sm100.cu) is the cost of its tcgen05 instructions: with a 128 x 16 A
// tile and N = 64 each takes 85 cycles where the arithmetic is 32, 5232 cycles per (query block, key block) pair, and its fp32
// dQ reductions are worth another 3200 of L2 time.  A pair shares the B operand, half of it in each CTA, so N = 128 runs at
// the arithmetic rate (2582 cycles for the five products); and a contraction over the pair's 256 keys halves the number of
// dQ tiles that are reduced.
//
// A pair owns 256 keys of one KV head, CTA r the r-th 128 of them, and visits every (query head of the GQA group, visible
// block of 128 queries).  Scores are transposed (keys on TMEM lanes), as in the single-CTA kernel:
//     S^T  = K Q^T            SS, 256x128x128    columns [0, 128)
//     dP^T = V dO^T           SS, 256x128x128    columns [128, 256)
//     P^T  = exp2(S^T c - lse2[q])               bf16 into columns [0, 32) and [96, 128)
//     dS^T = P^T o (dP^T - delta[q]) / sqrt(d)   bf16 into columns [128, 160) and [192, 224), and to shared memory: queries
//                                                [64 h, 64 h + 64) belong to CTA h, which so holds 64 queries x 256 keys
//     dV  += P^T dO           TS, 256x128x128    columns [256, 384)
//     dK  += dS^T Q           TS, 256x128x128    columns [384, 512)
//     dQ^T = K^T dS^T         SS, 128x128x256    columns [32, 96): CTA r gets head-dim rows [64 r, 64 r + 64); the second 64
//                                                query columns lie on the upper 64 lanes
// The tensor core runs dK_i-1, dP_i, dQ_i-1, dV_i, S_i+1.  The compute warps turn S_i into P_i while it works on the first three
// and dP_i into dS_i while it works on the last two; dQ_i-1 has the time of dK_i-1 and dP_i to get its operand from the other
// CTA, and the time of dV_i to leave the columns that S_i+1 takes.  Four warps of their own take it out of TMEM, through shared
// memory, and TMA adds it to memory (64 reductions per lane kept the SM's memory instructions queueing: 307 us against 291 below).
//
// 512 threads per CTA: warp 0 TMA, warp 1 MMA (the leader's issues for both), warp 2 exchange of dS, warps 4-7 dQ, warps 8-15
// compute (two per TMEM lane quarter, 64 query columns each).  Nobody orders global memory between the CTAs: a release at
// cluster scope waits for the SM's reductions in flight, 1800 cycles.  Shared memory: K and V (own keys), K of all 256 keys cut
// to the CTA's 64 head-dim columns, dS, dS on its way to the partner (one 16 KB bulk copy per block), dQ on its way to memory,
// and a ring of 16 KB tiles in the order in which the products want them: 64 rows of Q or dO for S^T and dP^T, 64 columns of
// them for dK and dV.
//
// What bounds it now is the chain of an iteration, 3600 cycles by clock marks: no unit is above 66 % busy (tensor pipe 65, shared
// memory and L1 63, issue 36).  The row statistics queue behind the tensor core's operand reads, so S_i -> P_i takes 1300 cycles, as
// long with its exp2 and conversions taken out; the exchange of dS takes 900 to 1600 of the 1030 that dK_i-1 and dP_i cover.
//
// Measured on B200, single-CTA kernel -> this one, us: 2 x 4096 tokens, 16 / 8 heads 362 -> 291; 16384, 16 / 8 2633 -> 2102 (1308
// TFLOP/s of the five causal products); 4096, 32 / 8 384 -> 281; 3 x 1408, 16 / 8 87 -> 71; 8 x 1024, 16 / 8 136 -> 117.
#include "attn_api.h"
#include "cta_pair.cuh"

namespace tb {

int make_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols);

namespace {

constexpr int HD = 128;
constexpr int TILE = 16384;               // 128 x 64 bf16
constexpr int RING = 4;
constexpr int STAT_BYTES = 1024;          // -lse2[128] | -delta*scale[128]
constexpr int BAR_BYTES = 256;
constexpr int SMEM_USED = (10 + RING) * TILE + 2 * STAT_BYTES + BAR_BYTES;
constexpr int SMEM_BYTES = 232448;        // the whole 227 KB: SMEM_USED plus alignment slack
static_assert(SMEM_USED <= SMEM_BYTES, "shared-memory plan exceeds the per-CTA limit");
constexpr int COMPUTE_WARPS = 8, DRAIN_WARPS = 4;
constexpr int NUM_THREADS = (4 + DRAIN_WARPS + COMPUTE_WARPS) * 32;
constexpr int COL_S = 0, COL_DP = 128, COL_DQ = 32, COL_DV = 256, COL_DK = 384;

struct Bars {
  // in the leader: announced by its producer with the bytes of both CTAs, or signalled by warps of both
  uint64_t k_full;
  uint64_t v_full;
  uint64_t full[RING];
  uint64_t s_read;          // one arrival per compute warp
  uint64_t p_ready;         // likewise
  uint64_t ds_ready;        // likewise
  uint64_t dq_drained;      // one per drain warp
  uint64_t ds_exchanged;    // the partner's ds_in has completed
  // in each CTA
  uint64_t empty[RING];     // the tensor core's
  uint64_t s_full;
  uint64_t dp_full;
  uint64_t dq_full;
  uint64_t acc_done;
  uint64_t ds_out;          // one arrival per compute warp whose queries are the partner's
  uint64_t ds_in;           // the partner's part of this CTA's queries is here
  uint64_t stat_full[2];
  uint32_t tmem_slot;
};
static_assert(sizeof(Bars) <= BAR_BYTES, "barrier block");

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// shared memory of this CTA to shared memory of the cluster
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t cluster_dst, const void* src, uint32_t bytes, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(cluster_dst),
               "r"(smem_u32(src)), "r"(bytes), "r"(cluster_bar)
               : "memory");
}

struct PairArgs {
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int64_t ld_dkv;
  const float* nds;    // [B, Hq, stat_stride]  -delta / sqrt(d)
  const float* nlse2;  // [B, Hq, stat_stride]  -lse * log2(e)
  int B, Sq, Skv, Hq, Hkv;
  int q_col0, k_col0, v_col0;
  int q_bstride, q_row0, kv_bstride, kv_row0, stat_stride, stat_row0;
  int kv_rows;       // rows of the k / v tensors: a load from there on reads zeros
  int causal;
  float scale, scale_log2;
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_bwd_2cta_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmQr, const __grid_constant__ CUtensorMap tmQc,
                     const __grid_constant__ CUtensorMap tmOr, const __grid_constant__ CUtensorMap tmOc,
                     const __grid_constant__ CUtensorMap tmDQ,
                     const __grid_constant__ PairArgs a, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  {
    uint32_t dyn;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if (static_cast<uint32_t>(smem - smem_raw) + SMEM_USED > dyn) {   // the same in both CTAs: nothing is set up yet
      if (threadIdx.x == 0) atomicCAS(err, 0, kErrAttnWait);
      return;
    }
  }
  uint8_t* sK = smem;                       // [head-dim half][128 keys x 128 B]
  uint8_t* sV = smem + 2 * TILE;
  uint8_t* sKT = smem + 4 * TILE;           // [256 keys x 128 B]: head-dim columns [64 r, 64 r + 64)
  uint8_t* sDS = smem + 6 * TILE;           // [256 keys x 128 B]: queries [64 r, 64 r + 64)
  uint8_t* sOut = smem + 8 * TILE;          // [128 keys x 128 B]: the partner's queries, on their way to it
  uint8_t* sDQ = smem + 9 * TILE;           // [drain warp][32 queries x 128 B]: 32 head-dim columns, on their way to memory
  uint8_t* sRing = smem + 10 * TILE;
  float* sStat = reinterpret_cast<float*>(sRing + RING * TILE);
  Bars* bars = reinterpret_cast<Bars*>(sRing + RING * TILE + 2 * STAT_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int nqb = a.Sq / 128, nkb = a.Skv / 128;
  const int ratio = a.Hq / a.Hkv;
  const int groups = a.B * a.Hkv;
  const int tile = static_cast<int>(blockIdx.x) >> 1;
  const int kpair = tile / groups;           // causal: pair 0 sees the most query blocks, it goes first
  const int g = tile % groups;
  const int kvh = g % a.Hkv, b = g / a.Hkv;
  const int kblk = 2 * kpair + rank;         // this CTA's key block
  const bool phantom = kblk >= nkb;          // an odd last block has a partner of zeros
  const int qb0 = a.causal ? 2 * kpair : 0;  // first query block that the pair sees
  const int n_qb = nqb - qb0;
  const int n_iter = n_qb * ratio;           // iteration = (query head of the group, query block)

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmQr);
    tma_prefetch_desc(&tmQc);
    tma_prefetch_desc(&tmOr);
    tma_prefetch_desc(&tmOc);
    tma_prefetch_desc(&tmDQ);
    mbar_init(&bars->k_full, 1);
    mbar_init(&bars->v_full, 1);
    for (int s = 0; s < RING; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->s_read, 2 * COMPUTE_WARPS);
    mbar_init(&bars->p_ready, 2 * COMPUTE_WARPS);
    mbar_init(&bars->ds_ready, 2 * COMPUTE_WARPS);
    mbar_init(&bars->dq_drained, 2 * DRAIN_WARPS);
    mbar_init(&bars->ds_exchanged, 1);
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->dq_full, 1);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->ds_out, COMPUTE_WARPS / 2);
    mbar_init(&bars->ds_in, 1);
    mbar_init(&bars->stat_full[0], 1);
    mbar_init(&bars->stat_full[1], 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_slot, 512);
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();   // the partner's barriers exist before anything is signalled on them
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_slot);

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      const uint32_t lead_k = map_to_cta(&bars->k_full, 0), lead_v = map_to_cta(&bars->v_full, 0);
      const uint32_t lead_full = map_to_cta(&bars->full[0], 0);
      const int kcol = a.k_col0 + kvh * HD, vcol = a.v_col0 + kvh * HD;
      const int pair_row = b * a.kv_bstride + a.kv_row0 + kpair * 256;
      const int row_1 = 2 * kpair + 1 < nkb ? pair_row + 128 : a.kv_rows;      // of the pair's second key block
      const int own_row = rank == 0 ? pair_row : row_1;
      if (rank == 0) {
        mbar_expect_tx(&bars->k_full, 2 * 2 * TILE);
        mbar_expect_tx(&bars->v_full, 2 * 4 * TILE);
      }
      tma_load_2d_pair(sK, &tmK, lead_k, kcol, own_row);
      tma_load_2d_pair(sK + TILE, &tmK, lead_k, kcol + 64, own_row);
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      // the next tile of the ring: `rows` takes 64 rows of 128 columns, else 128 rows of 64 columns
      auto load = [&](const CUtensorMap& map, int col, int row, bool rows) {
        if (!ok || !mbar_wait(&bars->empty[s], ph, err, kErrAttnWait)) { ok = false; return; }
        uint8_t* dst = sRing + s * TILE;
        const uint32_t bar = lead_full + 8 * s;
        if (rank == 0) mbar_expect_tx(&bars->full[s], 2 * TILE);
        if (rows) {
          tma_load_2d_pair(dst, &map, bar, col, row + 64 * rank);
          tma_load_2d_pair(dst + TILE / 2, &map, bar, col + 64, row + 64 * rank);
        } else {
          tma_load_2d_pair(dst, &map, bar, col + 64 * rank, row);
        }
        if (++s == RING) { s = 0; ph ^= 1; }
      };
      // where an iteration's operands lie; stepped along, since a division by the number of query blocks in front of every
      // load takes as many issue slots from the compute warps next to this one as they use themselves
      struct At { int qb, col, row; int64_t stat; };
      const int row0 = b * a.q_bstride + a.q_row0;
      const int64_t stat0 = (static_cast<int64_t>(b) * a.Hq + kvh * ratio) * a.stat_stride + a.stat_row0;
      auto step = [&](At x) {
        if (++x.qb == nqb) {
          x.qb = qb0;
          x.col += HD;
          x.row -= (n_qb - 1) * 128;
          x.stat += a.stat_stride - (n_qb - 1) * 128;
        } else {
          x.row += 128;
          x.stat += 128;
        }
        return x;
      };
      auto load_stats = [&](const At& x, int it) {
        float* dst = sStat + (it & 1) * (STAT_BYTES / 4);
        mbar_expect_tx(&bars->stat_full[it & 1], STAT_BYTES);
        bulk_load_1d(dst, a.nlse2 + x.stat, 512, &bars->stat_full[it & 1]);
        bulk_load_1d(dst + 128, a.nds + x.stat, 512, &bars->stat_full[it & 1]);
      };
      At now{qb0, kvh * ratio * HD, row0 + qb0 * 128, stat0 + qb0 * 128}, before = now;
      load(tmQr, a.q_col0 + now.col, now.row, true);
      load_stats(now, 0);
      tma_load_2d_pair(sV, &tmV, lead_v, vcol, own_row);
      tma_load_2d_pair(sV + TILE, &tmV, lead_v, vcol + 64, own_row);
      tma_load_2d_pair(sKT, &tmK, lead_v, kcol + 64 * rank, pair_row);
      tma_load_2d_pair(sKT + TILE, &tmK, lead_v, kcol + 64 * rank, row_1);
      if (n_iter > 1) load_stats(step(now), 1);
      for (int it = 0; it < n_iter && ok; ++it) {
        const At next = step(now);
        if (it > 0) load(tmQc, a.q_col0 + before.col, before.row, false);
        load(tmOr, now.col, now.row, true);
        // that tile's slot held the dP^T operand of iteration it - 1, whose product followed the one (dK of it - 2) that waited
        // for the last reads of the statistics of it - 2
        static_assert(RING == 4, "the statistics' buffer is free when the slot is");
        if (it > 1 && ok) load_stats(now, it);
        load(tmOc, now.col, now.row, false);
        if (it + 1 < n_iter) load(tmQr, a.q_col0 + next.col, next.row, true);
        before = now;
        now = next;
      }
      load(tmQc, a.q_col0 + before.col, before.row, false);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (leader only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc_st = make_idesc_bf16(256, 128, false, false);  // S^T, dP^T
      constexpr uint32_t idesc_acc = make_idesc_bf16(256, 128, false, true);  // dV, dK: A in TMEM, B MN-major
      constexpr uint32_t idesc_dq = make_idesc_bf16(128, 128, true, true);    // dQ^T: both MN-major
      const uint64_t dK = make_desc_sw128(smem_u32(sK), 16, 1024), dV = make_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t dKT = make_desc_sw128(smem_u32(sKT), TILE, 1024), dDS = make_desc_sw128(smem_u32(sDS), TILE, 1024);
      const uint64_t ring_k = make_desc_sw128(smem_u32(sRing), 16, 1024);     // K-major tiles: two halves of 8 KB
      const uint64_t ring_mn = make_desc_sw128(smem_u32(sRing), TILE, 1024);
      int slot = 0;
      uint32_t phase = 0;
      auto wait_full = [&]() { return mbar_wait(&bars->full[slot], phase, err, kErrAttnWait); };
      auto release = [&]() {
        umma2_commit_both(&bars->empty[slot]);
        if (++slot == RING) { slot = 0; phase ^= 1; }
      };
      auto scores = [&](uint32_t d, uint64_t da, uint64_t* done) {            // S^T or dP^T from the next tile
        const uint64_t db = ring_k + static_cast<uint64_t>(slot) * (TILE >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma2_f16_ss(tmem_base + d, da + (((ks >> 2) * TILE + (ks & 3) * 32) >> 4),
                       db + (((ks >> 2) * (TILE / 2) + (ks & 3) * 32) >> 4), idesc_st, ks != 0 ? 1u : 0u);
        umma2_commit_both(done);
        release();
      };
      // dV or dK from the next tile; the 64 queries of half h are the 32 columns from a_h on
      auto accumulate = [&](uint32_t d, uint32_t a0, uint32_t a1, bool first) {
        const uint64_t db = ring_mn + static_cast<uint64_t>(slot) * (TILE >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma2_f16_ts(tmem_base + d, tmem_base + (ks < 4 ? a0 : a1) + 8 * (ks & 3), db + ks * (2048 >> 4), idesc_acc,
                       (first && ks == 0) ? 0u : 1u);
        release();
      };
      auto query_gradient = [&](int it) {
        if (!mbar_wait(&bars->ds_in, it & 1, err, kErrAttnWait) || !mbar_wait(&bars->ds_exchanged, it & 1, err, kErrAttnWait))
          return false;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)
          umma2_f16_ss(tmem_base + COL_DQ, dKT + ks * (2048 >> 4), dDS + ks * (2048 >> 4), idesc_dq, ks != 0 ? 1u : 0u);
        umma2_commit_both(&bars->dq_full);
        return true;
      };
      // The tensor core takes its instructions in order: S_it+1 may follow dV_it, which reads P_it from the same columns, and
      // dP_it follow dK_it-1, which reads dS_it-1.
      bool ok = mbar_wait(&bars->k_full, 0, err, kErrAttnWait) && wait_full();
      if (ok) {
        tc_fence_after();
        scores(COL_S, dK, &bars->s_full);
        ok = mbar_wait(&bars->v_full, 0, err, kErrAttnWait);
      }
      for (int it = 0; it < n_iter && ok; ++it) {
        if (it > 0) {
          if (!wait_full() || !mbar_wait(&bars->ds_ready, (it - 1) & 1, err, kErrAttnWait)) { ok = false; break; }
          tc_fence_after();
          accumulate(COL_DK, COL_DP, COL_DP + 64, it == 1);
        }
        if (!wait_full()) { ok = false; break; }
        tc_fence_after();
        scores(COL_DP, dV, &bars->dp_full);
        if (it > 0) {                  // into columns of S_it between those that P_it takes
          if (!mbar_wait(&bars->s_read, it & 1, err, kErrAttnWait) || !query_gradient(it - 1)) { ok = false; break; }
        }
        if (!wait_full() || !mbar_wait(&bars->p_ready, it & 1, err, kErrAttnWait)) { ok = false; break; }
        tc_fence_after();
        accumulate(COL_DV, COL_S, COL_S + 96, it == 0);
        if (it > 0 && !mbar_wait(&bars->dq_drained, (it - 1) & 1, err, kErrAttnWait)) { ok = false; break; }
        if (it + 1 < n_iter) {
          if (!wait_full()) { ok = false; break; }
          tc_fence_after();
          scores(COL_S, dK, &bars->s_full);
        }
      }
      ok = ok && wait_full() && mbar_wait(&bars->ds_ready, (n_iter - 1) & 1, err, kErrAttnWait);
      if (ok) {
        tc_fence_after();
        accumulate(COL_DK, COL_DP, COL_DP + 64, n_iter == 1);
        ok = query_gradient(n_iter - 1);
      }
      if (ok) umma2_commit_both(&bars->acc_done);
    }
  } else if (warp == 2) {
    // ------------------------------------------------ exchange of dS^T between the CTAs
    if (elect_one()) {
      const uint32_t dst = map_to_cta(sDS + rank * TILE, rank ^ 1), dst_bar = map_to_cta(&bars->ds_in, rank ^ 1);
      const uint32_t lead_in = map_to_cta(&bars->ds_exchanged, 0);
      for (int it = 0; it < n_iter; ++it) {
        mbar_expect_tx(&bars->ds_in, TILE);
        if (!mbar_wait(&bars->ds_out, it & 1, err, kErrAttnWait)) break;
        bulk_copy_to_cta(dst, sOut, TILE, dst_bar);
        if (!mbar_wait(&bars->ds_in, it & 1, err, kErrAttnWait)) break;
        if (rank != 0) pair_arrive(lead_in);
      }
    }
  } else if (warp >= 4 && warp < 4 + DRAIN_WARPS) {
    // ------------------------------------------------ dQ^T from TMEM to memory
    const int quarter = warp & 3;
    const uint32_t t_dq = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + COL_DQ;
    const uint32_t lead_drained = map_to_cta(&bars->dq_drained, 0);
    uint8_t* const buf = sDQ + quarter * 4096;
    // this warp's part of the tile: a head-dim column per lane, 64 queries
    const int col = rank * 64 + (quarter & 1) * 32;
    int row = (b * a.Hq + kvh * ratio) * a.stat_stride + a.stat_row0 + (quarter >> 1) * 64;     // of the head's first query
    int qb = qb0;
    for (int it = 0; it < n_iter; ++it) {
      if (!mbar_wait_warp(&bars->dq_full, it & 1, err, kErrAttnWait)) break;
      tc_fence_after();
      uint32_t v[64];
      tmem_ld_32x32b_x32(t_dq, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
      tmem_ld_32x32b_x32(t_dq + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive(lead_drained);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (lane == 0) tma_wait_group_read<0>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j)          // one query's 32 columns are a row of 128 bytes
          *reinterpret_cast<uint32_t*>(buf + j * 128 + ((((lane >> 2) ^ (j & 7)) << 4) | ((lane & 3) << 2))) = v[32 * r + j];
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_reduce_add_2d(&tmDQ, buf, col, row + qb * 128 + r * 32);
          tma_commit_group();
        }
      }
      if (++qb == nqb) { qb = qb0; row += a.stat_stride; }
    }
    if (lane == 0) tma_wait_group<0>();
  } else if (warp >= 4 + DRAIN_WARPS) {
    // ------------------------------------------------ compute warps
    const int quarter = warp & 3;             // TMEM lane quarter this warp may touch
    const int half = (warp - 4 - DRAIN_WARPS) >> 2;     // which 64 of the block's 128 query columns
    const int row = quarter * 32 + lane;      // key inside the block
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t t_s = t_lane + COL_S + half * 64, t_p = t_lane + COL_S + half * 96, t_dp = t_lane + COL_DP + half * 64;
    const uint32_t lead_read = map_to_cta(&bars->s_read, 0), lead_p = map_to_cta(&bars->p_ready, 0);
    const uint32_t lead_ds = map_to_cta(&bars->ds_ready, 0);
    const float2 c2 = make_float2(a.scale_log2, a.scale_log2), sc2 = make_float2(a.scale, a.scale);
    uint8_t* const ds_row = (half == rank ? sDS + rank * TILE : sOut) + row * 128;     // 64 queries, 16-byte chunks swizzled
    bool ok = true;
    int qb = qb0;
    for (int it = 0; it < n_iter && ok; ++it) {
      const float* stat = sStat + (it & 1) * (STAT_BYTES / 4) + half * 64;
      // queries before the key are masked: the first `hidden` of this warp's columns (all of them for a key that is not there)
      const bool mask = phantom || (a.causal && qb <= kblk);
      const int hidden = phantom ? 64 : (kblk - qb) * 128 + row - half * 64;
      if (++qb == nqb) qb = qb0;
      if (!mbar_wait_warp(&bars->stat_full[it & 1], (it >> 1) & 1, err, kErrAttnWait) ||
          !mbar_wait_warp(&bars->s_full, it & 1, err, kErrAttnWait)) { ok = false; break; }
      tc_fence_after();
      uint32_t p[64];                         // P^T in fp32, kept until dS^T
      tmem_ld_32x32b_x32(t_s, *reinterpret_cast<uint32_t(*)[32]>(&p[0]));
      tmem_ld_32x32b_x32(t_s + 32, *reinterpret_cast<uint32_t(*)[32]>(&p[32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive(lead_read);
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[8];
#pragma unroll
        for (int i = 16 * c; i < 16 * c + 16; i += 4) {
          const float4 nl = *reinterpret_cast<const float4*>(stat + i);          // -lse2 of four queries
          const float2 t0 = fma2(make_float2(__uint_as_float(p[i]), __uint_as_float(p[i + 1])), c2, make_float2(nl.x, nl.y));
          const float2 t1 = fma2(make_float2(__uint_as_float(p[i + 2]), __uint_as_float(p[i + 3])), c2, make_float2(nl.z, nl.w));
          float e[4] = {ex2(t0.x), ex2(t0.y), ex2(t1.x), ex2(t1.y)};
          if (mask) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (i + k < hidden) e[k] = 0.f;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) p[i + k] = __float_as_uint(e[k]);
          pk[(i - 16 * c) / 2] = pack_bf16x2(e[0], e[1]);
          pk[(i - 16 * c) / 2 + 1] = pack_bf16x2(e[2], e[3]);
        }
        tmem_st_32x32b_x8(t_p + 8 * c, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive(lead_p);
      if (!mbar_wait_warp(&bars->dp_full, it & 1, err, kErrAttnWait)) { ok = false; break; }
      tc_fence_after();
      uint32_t pd[32];
#pragma unroll
      for (int c = 0; c < 4; ++c) {           // dS^T goes where dP^T has been read already
        uint32_t dp[16];
        tmem_ld_32x32b_x16(t_dp + 16 * c, dp);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const int at = 16 * c + i;
          const float4 nd = *reinterpret_cast<const float4*>(stat + 128 + at);    // -delta * scale
          const float2 u0 = fma2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), sc2, make_float2(nd.x, nd.y));
          const float2 u1 = fma2(make_float2(__uint_as_float(dp[i + 2]), __uint_as_float(dp[i + 3])), sc2, make_float2(nd.z, nd.w));
          const float2 d0 = mul2(make_float2(__uint_as_float(p[at]), __uint_as_float(p[at + 1])), u0);
          const float2 d1 = mul2(make_float2(__uint_as_float(p[at + 2]), __uint_as_float(p[at + 3])), u1);
          pd[at / 2] = pack_bf16x2(d0.x, d0.y);
          pd[at / 2 + 1] = pack_bf16x2(d1.x, d1.y);
        }
        tmem_st_32x32b_x8(t_dp + 8 * c, *reinterpret_cast<const uint32_t(*)[8]>(&pd[8 * c]));
      }
      // the tensor core and the copy to the partner have read the dS^T tiles of the iteration before
      if (it > 0 && !mbar_wait_warp(&bars->dq_full, (it - 1) & 1, err, kErrAttnWait)) { ok = false; break; }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(ds_row + ((j ^ (row & 7)) << 4)) = make_uint4(pd[4 * j], pd[4 * j + 1], pd[4 * j + 2], pd[4 * j + 3]);
      tmem_st_wait();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (half != rank) mbar_arrive(&bars->ds_out);
        pair_arrive(lead_ds);
      }
    }
    if (ok && mbar_wait_warp(&bars->acc_done, 0, err, kErrAttnWait) && !phantom) {
      // warps of half 0 write dV, of half 1 dK: one key row per lane
      tc_fence_after();
#pragma unroll 1
      for (int col = 0; col < HD; col += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(t_lane + COL_DV + half * 128 + col, v);
        tmem_ld_wait();
        __nv_bfloat16* dst = (half == 0 ? a.dv : a.dk) + (static_cast<int64_t>(b) * a.Skv + kblk * 128 + row) * a.ld_dkv + kvh * HD + col;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 pk;
          pk.x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
          pk.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
          pk.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
          pk.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
          *reinterpret_cast<uint4*>(dst + 8 * j) = pk;
        }
      }
    }
  }

  if (*reinterpret_cast<volatile int*>(err) != 0) {
    // a wait expired somewhere: give copies and MMAs in flight time to land before TMEM is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // neither CTA retires while its partner may still signal its barriers or read its operands
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

// Same contract as attn_bwd_fused, which checks the arguments and decides.
int attn_bwd_2cta(const AttnOperand& q, const AttnOperand& k, const AttnOperand& v, const void* d_o, float* dq_acc, void* dk,
                  void* dv, int64_t ld_dkv, const float* nds, const float* nlse2, int B, int Sq, int Skv, int Hq, int Hkv,
                  bool causal, int* err, cudaStream_t stream, const AttnPairLayout& lay) {
  const uint64_t Mq = static_cast<uint64_t>(lay.q_rows), Mk = static_cast<uint64_t>(lay.kv_rows);
  const uint64_t ld_o = static_cast<uint64_t>(Hq) * HD;
  CUtensorMap tk, tv, tqr, tqc, tor, toc, tdq;
  int r = make_tmap_2d(&tk, k.ptr, 2, Mk, k.ld, k.ld, 128, 64);
  if (r) return r - 100;
  r = make_tmap_2d(&tv, v.ptr, 2, Mk, v.ld, v.ld, 128, 64);
  if (r) return r - 200;
  r = make_tmap_2d(&tqr, q.ptr, 2, Mq, q.ld, q.ld, 64, 64);
  if (!r) r = make_tmap_2d(&tqc, q.ptr, 2, Mq, q.ld, q.ld, 128, 64);
  if (r) return r;
  r = make_tmap_2d(&tor, d_o, 2, Mq, ld_o, ld_o, 64, 64);
  if (!r) r = make_tmap_2d(&toc, d_o, 2, Mq, ld_o, ld_o, 128, 64);
  if (r) return r - 300;
  r = make_tmap_2d(&tdq, dq_acc, 4, static_cast<uint64_t>(B) * Hq * lay.stat_stride, HD, HD, 32, 32);
  if (r) return r - 400;
  PairArgs a{};
  a.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  a.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  a.ld_dkv = ld_dkv;
  a.nds = nds;
  a.nlse2 = nlse2;
  a.B = B; a.Sq = Sq; a.Skv = Skv; a.Hq = Hq; a.Hkv = Hkv;
  a.q_col0 = static_cast<int>(q.col0);
  a.k_col0 = static_cast<int>(k.col0);
  a.v_col0 = static_cast<int>(v.col0);
  a.q_bstride = lay.q_bstride; a.q_row0 = lay.q_row0; a.kv_bstride = lay.kv_bstride; a.kv_row0 = lay.kv_row0;
  a.stat_stride = lay.stat_stride; a.stat_row0 = lay.stat_row0;
  a.kv_rows = static_cast<int>(lay.kv_rows);
  a.causal = causal ? 1 : 0;
  a.scale = 1.f / sqrtf(static_cast<float>(HD));
  a.scale_log2 = a.scale * 1.4426950408889634f;
  if (!ensure_dynamic_smem(reinterpret_cast<const void*>(attn_bwd_2cta_kernel), SMEM_BYTES)) return -20;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * ((Skv / 128 + 1) / 2) * B * Hkv);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, attn_bwd_2cta_kernel, tk, tv, tqr, tqc, tor, toc, tdq, a, err) == cudaSuccess ? 0 : -21;
}

}  // namespace tb
