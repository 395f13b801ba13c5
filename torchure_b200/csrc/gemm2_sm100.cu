// bf16 GEMM on CTA PAIRS (tcgen05.mma.cta_group::2): two CTAs of a cluster, on two SMs, compute one 256 x 256 output
// tile.  Each CTA brings its own 128 rows of A and HALF of the 256 rows of B into its shared memory; one
// instruction, issued by the leader CTA, runs both tensor cores on 256 x 256 x 16, each reading the other half of B
// from its partner.  A single CTA with a 128 x 256 tile fetches 12 KB of operands per k-step of 16 and measures 160
// cycles for it on B200 (128 would be the arithmetic); the pair fetches 8 KB per CTA and measures 128.
//
//   per CTA: 6 pipeline stages of 32 KB (A 128 x 64, B 128 x 64), 192 threads:
//     warp 0      TMA producer: its A rows and its half of B, completing on the LEADER's "full" barrier (which the
//                 leader's producer arms with the byte count of both CTAs)
//     warp 1      TMEM allocator; in the leader also the MMA issuer.  tcgen05.commit with a cluster mask releases the
//                 stage in both CTAs ("empty") and hands the accumulator to both epilogues ("tfull")
//     warps 2..5  epilogue of this CTA's 128 rows (TMEM lanes), as in the single-CTA kernel; both CTAs' epilogue
//                 threads arrive on the leader's "tempty" barrier
//   Two 256-column accumulators per CTA: the epilogue of tile i overlaps the main loop of tile i + 1.
//
// Operand layouts, output modes (bf16 store, fp32 store, fp32 reduce-add) and split-K are those of the single-CTA
// kernel in gemm_sm100.cu, which remains the path of the fused GEMM + collective kernels and of wide products of at most
// 128 rows; problems with few tiles run on gemm_small_sm100.cu (the choice is gemm_plan in gemm_sm100.cu).
// Every wait is bounded; the two CTAs meet at a cluster barrier before anyone touches a partner's barrier and again
// before either releases its tensor memory.
#include "api.h"
#include "cta_pair.cuh"

#include <type_traits>

namespace tb {

int make_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols);

namespace {

constexpr int BM = 128;            // rows of A (and of the output) per CTA
constexpr int BN = 256;            // output columns of the pair's tile
constexpr int BNH = BN / 2;        // rows of B held by one CTA
constexpr int BK = 64, STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;             // 16 KB
constexpr int B_BYTES = BNH * BK * 2;            // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;   // 32 KB
constexpr int EPI_BUF = 4096;                    // 32 rows x 128 B
constexpr int EPI_BYTES = 4 * 2 * EPI_BUF;
constexpr int BAR_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + BAR_BYTES + 1024;
constexpr int NUM_THREADS = 192;
constexpr uint32_t TMEM_COLS = 512;

// What the epilogue does beside storing the tile.
//   kEpiStore   nothing
//   kEpiSwiglu  the tile's left half holds 128 gate columns, the right half the up columns of the same units (the leader's B
//               rows come from the gate block of W, the partner's from the up block, F rows further down): both are
//               stored as they are (when wanted) and silu(gate) * up goes to a third matrix.  Both factors are rounded to
//               bf16 first, as a pass over the stored matrix would see them.
//   kEpiCe      instead of the tile every row leaves (maximum, sum of exponentials relative to it) of its columns, taken from
//               the values rounded to bf16, and the logit of its label if that lies in the tile: the loss of a pass without
//               gradients then needs no logits in memory.  (With the tile stored as well, to spare the softmax pass of a
//               training step its first read, the product lost what that pass gained: 4096 x 151936 x 1024 834 + 543 us
//               before, 906 + 436 with; 4096 x 128256 x 2048 1305 + 478 before, 1416 + 420 with.)
//   kEpiSwigluBwd  the tile is d(act); the stored gate and up values of the same elements are read (32 columns at a time, the
//               next ones while the present ones are worked on) and d(gate), d(up) are stored instead of it.
enum { kEpiStore = 0, kEpiSwiglu = 1, kEpiCe = 2, kEpiSwigluBwd = 3 };

struct EpiArgs {
  int store;               // kEpiSwiglu: write gate and up
  const int64_t* labels;   // kEpiCe: [M], out of range: no target
  float2* stats;           // kEpiCe: [tiles along N][M]
  float* target;           // kEpiCe: [M]
  const __nv_bfloat16* gu; // kEpiSwigluBwd: [M, 2N], N a multiple of 16, 32-byte aligned
};

// 16 bf16 values, one 32-byte sector
__device__ __forceinline__ void load_sector(const void* p, uint32_t* r) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p));
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// N: columns of C; for kEpiSwiglu the F columns of one half (W has 2F rows)
template <bool A_MN, bool B_MN, int OUT, int EPI>
__device__ __forceinline__ void
gemm2_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmUp,
           const CUtensorMap& tmAct, const EpiArgs& ea, int M, int N, int K, int splits, int slice_rows, int group, int* err) {
  constexpr int TN = EPI == kEpiSwiglu ? BNH : BN;   // columns of C per tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint8_t* epi = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + EPI_BYTES);
  uint64_t* full = bars;                     // [STAGES]  used in the leader
  uint64_t* empty = bars + STAGES;           // [STAGES]  one per CTA
  uint64_t* tfull = bars + 2 * STAGES;       // [2]       one per CTA
  uint64_t* tempty = bars + 2 * STAGES + 2;  // [2]       used in the leader
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();           // 0: leader
  const int cluster = static_cast<int>(blockIdx.x) >> 1;
  const int num_clusters = static_cast<int>(gridDim.x) >> 1;
  const int num_m = (M + 2 * BM - 1) / (2 * BM);
  const int num_n = (N + TN - 1) / TN;
  const int num_tiles = num_m * num_n;
  const int num_kb = (K + BK - 1) / BK;
  // split-K: work unit u = (tile u % num_tiles, K slice u / num_tiles); slices add into C with TMA reduce-add
  const int num_units = num_tiles * splits;
  const int kb_per = (num_kb + splits - 1) / splits;
  // Tiles go down the columns, one column of tiles after the other, or (gemm2_bf16) down `group` rows of tiles at a time, through
  // all columns.
  auto place = [&](int tile, int& tm, int& tn) {
    if (EPI == kEpiStore && group > 0) {
      const int g0 = tile / (group * num_n) * group;
      const int rows = min(group, num_m - g0), at = tile - g0 * num_n;
      tm = g0 + at % rows;
      tn = at / rows;
    } else {
      tm = tile % num_m;
      tn = tile / num_m;
    }
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);      // the leader's producer arrives, announcing the bytes of both CTAs
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 256);  // the epilogue threads of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();   // the partner's barriers exist before anything is signalled on them
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t lead_full_addr[STAGES];
#pragma unroll
      for (int s = 0; s < STAGES; ++s) lead_full_addr[s] = map_to_cta(&full[s], 0);
      for (int unit = cluster; unit < num_units && ok; unit += num_clusters) {
        const int tile = unit % num_tiles;
        const int kb0 = (unit / num_tiles) * kb_per;
        const int kb1 = min(num_kb, kb0 + kb_per);
        int tm, tn;
        place(tile, tm, tn);
        const int m0 = tm * 2 * BM + static_cast<int>(rank) * BM;
        // the leader holds the first 128 B rows of the tile
        const int n0 = tn * TN + static_cast<int>(rank) * (EPI == kEpiSwiglu ? N : BNH);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, err, kErrProducerEmptyWait)) { ok = false; break; }
          uint8_t* sA = smem + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          // Only the leader arms its barrier, with the byte count of both CTAs: the partner's copies may well land
          // first (the pending count then dips below zero until the leader's announcement arrives), and a remote
          // arrival per stage would put a cluster-scope release on the producer's critical path.
          const uint32_t lead_full = lead_full_addr[stage];
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * STAGE_BYTES);
          const int k0 = kb * BK;
          if (!A_MN) {
            tma_load_2d_pair(sA, &tmA, lead_full, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sA + j * 8192, &tmA, lead_full, m0 + j * 64, k0);
          }
          if (!B_MN) {
            tma_load_2d_pair(sB, &tmB, lead_full, k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(sB + j * 8192, &tmB, lead_full, n0 + j * 64, k0);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader only) ------------------
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      constexpr uint32_t a_lbo = A_MN ? 8192u : 16u, b_lbo = B_MN ? 8192u : 16u;
      constexpr uint32_t a_step = A_MN ? (2048u >> 4) : (32u >> 4);  // descriptor advance per k=16
      constexpr uint32_t b_step = B_MN ? (2048u >> 4) : (32u >> 4);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int unit = cluster; unit < num_units && ok; unit += num_clusters) {
        const int kb0 = (unit / num_tiles) * kb_per;
        const int kb1 = min(num_kb, kb0 + kb_per);
        if (kb0 >= kb1) continue;  // empty K slice: every role skips it
        const int acc = it & 1;
        if (!mbar_wait(&tempty[acc], ((it >> 1) & 1) ^ 1, err, kErrMmaTmemEmptyWait)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full[stage], phase, err, kErrMmaFullWait)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * STAGE_BYTES);
          const uint64_t da = make_desc_sw128(a_addr, a_lbo, 1024);
          const uint64_t db = make_desc_sw128(a_addr + A_BYTES, b_lbo, 1024);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            umma2_f16_ss(d_tmem, da + static_cast<uint64_t>(k * a_step), db + static_cast<uint64_t>(k * b_step), idesc,
                         (kb != kb0 || k != 0) ? 1u : 0u);
          }
          umma2_commit_both(&empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma2_commit_both(&tfull[acc]);
        ++it;
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ----------------------
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    uint8_t* buf0 = epi + q * 2 * EPI_BUF;
    constexpr int COLS = (OUT == 0) ? 64 : 32;  // columns per staged slab (128 B per row)
    int it = 0;
    int slab = 0;
    bool ok = true;
    for (int unit = cluster; unit < num_units && ok; unit += num_clusters) {
      const int tile = unit % num_tiles;
      if ((unit / num_tiles) * kb_per >= num_kb) continue;  // empty K slice
      const int c_row = (unit / num_tiles) * slice_rows;    // each slice has rows of its own in a workspace
      int tm, tn;
      place(tile, tm, tn);
      const int m0 = tm * 2 * BM + static_cast<int>(rank) * BM;
      const int n0 = tn * TN;
      const int acc = it & 1;
      if constexpr (EPI == kEpiStore) {
        // In a branch of its own down to the wait: code of the other epilogues in the same loop body, never run here, cost the
        // plain bf16 store 2 - 7 % of a short product (8192 x 3072 x 64 24.3 against 22.8 us, 1536 x 6144 x 256 13.55
        // against 13.0).
        if (!mbar_wait_warp(&tfull[acc], (it >> 1) & 1, err, kErrEpilogueTmemFullWait)) { ok = false; break; }
        tc_fence_after();
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
        const bool rows_live = (m0 + q * 32) < M;
        const uint32_t lead_tempty = map_to_cta(&tempty[acc], 0);
#pragma unroll 1
        for (int c = 0; c < BN / COLS; ++c) {
          uint32_t v[64];
          __syncwarp();      // one lane stored the slab before
          if (OUT == 0) {
            tmem_ld_32x32b_x32(t_row + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
            tmem_ld_32x32b_x32(t_row + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
          } else {
            tmem_ld_32x32b_x32(t_row + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
          }
          tmem_ld_wait();
          if (c == BN / COLS - 1) {
            // the accumulator is in registers: hand it back to the leader's MMA warp
            tc_fence_before();
            remote_arrive(lead_tempty);
          }
          if (rows_live && (n0 + c * COLS) < N) {
            uint8_t* buf = buf0 + (slab & 1) * EPI_BUF;
            ++slab;
            if (lane == 0) tma_wait_group_read<1>();  // the store that last used this buffer has read it
            __syncwarp();
            uint8_t* row = buf + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint4 pk;
              if (OUT == 0) {
                pk.x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
                pk.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
                pk.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
                pk.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
              } else {
                pk.x = v[4 * j + 0]; pk.y = v[4 * j + 1]; pk.z = v[4 * j + 2]; pk.w = v[4 * j + 3];
              }
              *reinterpret_cast<uint4*>(row + ((j ^ (lane & 7)) << 4)) = pk;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (OUT == 2) tma_reduce_add_2d(&tmC, buf, n0 + c * COLS, m0 + q * 32);
              else tma_store_2d(&tmC, buf, n0 + c * COLS, c_row + m0 + q * 32);
              tma_commit_group();
            }
          }
        }
      } else {
        uint32_t gv[2][16], uv[2][16];     // kEpiSwigluBwd: gate and up of 32 columns, two sets
        auto load_gu = [&](int c, auto set_tag) {     // half `set` of slab c of this lane's row; zeros outside the matrix
          constexpr int set = decltype(set_tag)::value;
          const int gr = m0 + q * 32 + lane;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int col = n0 + c * 64 + set * 32 + j * 16;
            const bool in = gr < M && col < N;
            const __nv_bfloat16* p = ea.gu + static_cast<int64_t>(gr) * 2 * N + col;
            if (in) {
              load_sector(p, &gv[set][8 * j]);
              load_sector(p + N, &uv[set][8 * j]);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) gv[set][8 * j + i] = uv[set][8 * j + i] = 0u;
            }
          }
        };
        if constexpr (EPI == kEpiSwigluBwd) {
          load_gu(0, std::integral_constant<int, 0>{});
          load_gu(0, std::integral_constant<int, 1>{});
        }
        if (!mbar_wait_warp(&tfull[acc], (it >> 1) & 1, err, kErrEpilogueTmemFullWait)) { ok = false; break; }
        tc_fence_after();
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
        const bool rows_live = (m0 + q * 32) < M;
        const uint32_t lead_tempty = map_to_cta(&tempty[acc], 0);
        // 32 rows x 128 bytes of packed output, one row per lane, to columns `col` of a matrix
        auto emit = [&](const uint32_t (&pk)[32], const CUtensorMap& tm, int col) {
          uint8_t* buf = buf0 + (slab & 1) * EPI_BUF;
          ++slab;
          if (lane == 0) tma_wait_group_read<1>();  // the store that last used this buffer has read it
          __syncwarp();
          uint8_t* row = buf + lane * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(row + ((j ^ (lane & 7)) << 4)) = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tm, buf, col, m0 + q * 32);
            tma_commit_group();
          }
        };
        if constexpr (EPI == kEpiSwiglu) {
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            uint32_t pg[32], pu[32], pa[32];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              uint32_t g[32], u[32];
              __syncwarp();
              tmem_ld_32x32b_x32(t_row + c * 64 + hf * 32, g);
              tmem_ld_32x32b_x32(t_row + BNH + c * 64 + hf * 32, u);
              tmem_ld_wait();
              if (c == 1 && hf == 1) {
                tc_fence_before();
                remote_arrive(lead_tempty);
              }
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const uint32_t gp = pack_bf16x2(__uint_as_float(g[2 * i]), __uint_as_float(g[2 * i + 1]));
                const uint32_t up = pack_bf16x2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
                const float gx = __uint_as_float(gp << 16), gy = __uint_as_float(gp & 0xffff0000u);
                const float ux = __uint_as_float(up << 16), uy = __uint_as_float(up & 0xffff0000u);
                pg[hf * 16 + i] = gp;
                pu[hf * 16 + i] = up;
                pa[hf * 16 + i] = pack_bf16x2(__fdividef(gx, 1.f + __expf(-gx)) * ux, __fdividef(gy, 1.f + __expf(-gy)) * uy);
              }
            }
            if (rows_live && (n0 + c * 64) < N) {
              emit(pa, tmAct, n0 + c * 64);
              if (ea.store) {
                emit(pg, tmC, n0 + c * 64);
                emit(pu, tmUp, n0 + c * 64);
              }
            }
          }
        } else if constexpr (EPI == kEpiSwigluBwd) {
#pragma unroll 1
          for (int c = 0; c < BN / 64; ++c) {
            uint32_t pg[32], pu[32];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              uint32_t d[32];
              __syncwarp();
              tmem_ld_32x32b_x32(t_row + c * 64 + hf * 32, d);
              tmem_ld_wait();
              if (c == BN / 64 - 1 && hf == 1) {
                tc_fence_before();
                remote_arrive(lead_tempty);
              }
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const uint32_t gp = gv[hf][i], up = uv[hf][i];
                const float gx = __uint_as_float(gp << 16), gy = __uint_as_float(gp & 0xffff0000u);
                const float ux = __uint_as_float(up << 16), uy = __uint_as_float(up & 0xffff0000u);
                const float ex = __uint_as_float(d[2 * i]), ey = __uint_as_float(d[2 * i + 1]);
                const float sx = __fdividef(1.f, 1.f + __expf(-gx)), sy = __fdividef(1.f, 1.f + __expf(-gy));
                // d silu(g)/dg = s (1 + g (1 - s))
                pg[hf * 16 + i] = pack_bf16x2(ex * ux * sx * (1.f + gx * (1.f - sx)), ey * uy * sy * (1.f + gy * (1.f - sy)));
                pu[hf * 16 + i] = pack_bf16x2(ex * gx * sx, ey * gy * sy);
              }
              if (c < BN / 64 - 1) {
                if (hf == 0) load_gu(c + 1, std::integral_constant<int, 0>{});
                else load_gu(c + 1, std::integral_constant<int, 1>{});
              }
            }
            if (rows_live && (n0 + c * 64) < N) {
              emit(pg, tmC, n0 + c * 64);
              emit(pu, tmUp, n0 + c * 64);
            }
          }
        } else {
          // kEpiCe: running maximum and sum of this lane's row over the tile's columns
          float ce_m = -INFINITY, ce_s = 0.f;
          const int ce_row = m0 + q * 32 + lane;
          int64_t ce_label = -1;
          if (ce_row < M) ce_label = ea.labels[ce_row];
#pragma unroll 1
          for (int c = 0; c < BN / COLS; ++c) {
            uint32_t v[64];
            __syncwarp();    // the lane that holds the label took longer
            tmem_ld_32x32b_x32(t_row + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
            tmem_ld_32x32b_x32(t_row + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
            tmem_ld_wait();
            if (c == BN / COLS - 1) {
              // the accumulator is in registers: hand it back to the leader's MMA warp
              tc_fence_before();
              remote_arrive(lead_tempty);
            }
            if (rows_live && (n0 + c * COLS) < N) {
              constexpr float kLog2e = 1.4426950408889634f;
              const int left = N - (n0 + c * COLS);      // live columns of this slab (64 or more: all)
              float lm = -INFINITY;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                // from here on the rounded values; columns past the end count as -inf
                const uint32_t xy = pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                float x = __uint_as_float(xy << 16), y = __uint_as_float(xy & 0xffff0000u);
                if (left < COLS) {
                  if (2 * i >= left) x = -INFINITY;
                  if (2 * i + 1 >= left) y = -INFINITY;
                }
                v[2 * i] = __float_as_uint(x);
                v[2 * i + 1] = __float_as_uint(y);
                lm = fmaxf(lm, fmaxf(x, y));
              }
              if (lm > ce_m) { ce_s *= ex2_approx((ce_m - lm) * kLog2e); ce_m = lm; }
              // 2^(x log2 e + nm) per column, nm = -max log2 e rounded; what the rounding took, the same for every column, is given
              // back to their sum (0: only -inf so far, they add nothing)
              const float nm = ce_m == -INFINITY ? 0.f : -ce_m * kLog2e;
              const float left_out = ce_m == -INFINITY ? 0.f : fmaf(-ce_m, kLog2e, -nm);
              float s0 = 0.f, s1 = 0.f;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                s0 += ex2_approx(fmaf(__uint_as_float(v[2 * i]), kLog2e, nm));
                s1 += ex2_approx(fmaf(__uint_as_float(v[2 * i + 1]), kLog2e, nm));
              }
              ce_s += fmaf(s0 + s1, left_out * 0.6931471805599453f, s0 + s1);
              const int64_t at = ce_label - (n0 + c * COLS);
              if (at >= 0 && at < COLS && at < left) {
                float t = 0.f;
#pragma unroll
                for (int i = 0; i < 64; ++i)
                  if (at == i) t = __uint_as_float(v[i]);
                ea.target[ce_row] = t;
              }
            }
          }
          if (ce_row < M) ea.stats[static_cast<int64_t>(tn) * M + ce_row] = make_float2(ce_m, ce_s);
        }
      }
      ++it;
    }
    if (lane == 0) tma_wait_group<0>();
  }

  // ------------------------------ teardown ------------------------------------
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
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <bool A_MN, bool B_MN, int OUT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmC, int M, int N, int K, int splits, int slice_rows, int group, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  gemm2_body<A_MN, B_MN, OUT, kEpiStore>(tmA, tmB, tmC, tmC, tmC, EpiArgs{}, M, N, K, splits, slice_rows, group, err);
}

// Measured on B200, M x F x K, product + pass over it before, fused now, fused without storing gate and up: 8192 x 3072 x 1024
// 98.7, 80.1, 70.4 us; 8192 x 8192 x 2048 411, 370, 341; 2048 x 3072 x 1024 33.0, 25.9, 23.2; 8192 x 1024 x 256 29.4, 23.3,
// 19.9.  The epilogue (two special-function operations per unit and 1.5 times the stores) hides behind the k loop.
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2_swiglu_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmGate, const __grid_constant__ CUtensorMap tmUp,
                    const __grid_constant__ CUtensorMap tmAct, const __grid_constant__ EpiArgs ea, int M, int F, int K,
                    int* err) {
  pdl_wait();
  pdl_launch_dependents();
  gemm2_body<false, false, 0, kEpiSwiglu>(tmA, tmB, tmGate, tmUp, tmAct, ea, M, F, K, 1, 0, 0, err);
}

// Bound by its epilogue when K is short: 256 columns of two special-function operations, two loads and two stores per row
// against K / 64 x 512 cycles of products; and the last wave's epilogue has no products to hide behind.  It spares the passes
// over d(act).  gemm2_swiglu_bwd_pays has the rule.
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2_swiglu_bwd_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmGate, const __grid_constant__ CUtensorMap tmUp,
                        const __grid_constant__ EpiArgs ea, int M, int F, int K, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  gemm2_body<false, true, 0, kEpiSwigluBwd>(tmA, tmB, tmGate, tmUp, tmGate, ea, M, F, K, 1, 0, 0, err);
}

// Measured on B200, against the product and a loss pass over its output: 4096 x 151936 x 1024 834 + 238 us before, 773 + 17
// now; 1024 x 50257 x 512 73 + 25 before, 75 + 7 now.
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2_ce_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ EpiArgs ea, int M, int N, int K, int* err) {
  pdl_wait();
  pdl_launch_dependents();
  gemm2_body<false, false, 0, kEpiCe>(tmA, tmB, tmB, tmB, tmB, ea, M, N, K, 1, 0, 0, err);
}

// How many CTA pairs the device can hold at once.  The two CTAs of a pair sit on the two SMs of one TPC; a part with
// TPCs of which one SM is fused off holds fewer pairs than SMs / 2.  The persistent schedule hands work to exactly this
// many pairs: a pair that had to wait for a free TPC would start a whole problem late.
int g_pair_capacity = 0;

template <class... Params, class... Args>
int launch_pairs(void (*kern)(Params...), int units, int num_sms, cudaStream_t stream, Args... args) {
  if (!ensure_dynamic_smem(reinterpret_cast<const void*>(kern), SMEM_BYTES)) return -20;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  if (g_pair_capacity == 0) {
    int dev = 0, all_sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&all_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return -23;
    cfg.gridDim = dim3(2 * (all_sms / 2));
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) return -23;
    g_pair_capacity = n < all_sms / 2 ? n : all_sms / 2;
  }
  const int pairs = g_pair_capacity < num_sms / 2 ? g_pair_capacity : num_sms / 2;    // num_sms: without the reserved ones
  const int clusters = units < pairs ? units : pairs;
  cfg.gridDim = dim3(2 * clusters);
  cfg.stream = stream;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess ? 0 : -21;
}

}  // namespace

int gemm_pair_capacity() { return g_pair_capacity; }

// Same contract as gemm_bf16 (gemm_sm100.cu), which decides between this kernel and the others (gemm_plan).
int gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
               bool a_mn, bool b_mn, int out_mode, int splits, int* err, int num_sms, cudaStream_t stream,
               int64_t slice_rows) {
  CUtensorMap ta, tb_, tc;
  int r;
  // K-major operand [R, K]: box 64 (k) x tile rows.  MN-major operand stored [K, R]: box 64 (r) x 64 (k rows).
  r = a_mn ? make_tmap_2d(&ta, A, 2, K, M, lda, 64, 64) : make_tmap_2d(&ta, A, 2, M, K, lda, BM, 64);
  if (r) return r;
  r = b_mn ? make_tmap_2d(&tb_, B, 2, K, N, ldb, 64, 64) : make_tmap_2d(&tb_, B, 2, N, K, ldb, BNH, 64);
  if (r) return r - 100;
  // slices with rows of their own: the padding rows up to slice_rows take what the ragged last tile stores
  const uint64_t c_rows = slice_rows > 0 ? static_cast<uint64_t>(slice_rows) * splits : M;
  r = out_mode == 0 ? make_tmap_2d(&tc, C, 2, c_rows, N, ldc, 32, 64) : make_tmap_2d(&tc, C, 4, c_rows, N, ldc, 32, 32);
  if (r) return r - 200;
  // The order of the tiles, so that the clusters in flight cover a block of the output as square as can be and read A and B from
  // memory once: a wide output column by column of tiles (all rows at a time), a tall one by groups of as many rows of tiles as one
  // wave holds of whole rows.  Column by column a tall output read A once per column of tiles: the gradient of a head its 1.2 GB of
  // logits four times.  Measured on B200, cold inputs, M x N x K, column by column, in groups, us: weight gradients 151936 x 1024 x 1024
  // 307, 243; 19456 x 2560 x 4096 328, 264; 16384 x 2048 x 8192 408, 350; 50257 x 512 x 600 48.0, 43.6; bf16 16384 x 1024 x 2048
  // 57.4, 52.9; 8192 x 2048 x 16384 388, 365; 8192 x 1024 x 3072 43.7, 41.6; wide ones, in groups slower: 2560 x 9728 x 4096 140, 149;
  // 2048 x 8192 x 8192 180, 189; 4096 x 6144 x 2560 87.8, 88.8; about square, 8192 x 8192 x 2048, no difference.
  const int pairs = g_pair_capacity > 0 && g_pair_capacity < num_sms / 2 ? g_pair_capacity : num_sms / 2;
  const int num_m = (M + 2 * BM - 1) / (2 * BM), num_n = (N + BN - 1) / BN;
  const int units = num_m * num_n * splits;
  const int group = splits == 1 && num_n > 1 && num_m > num_n ? (pairs > 4 * num_n ? pairs / num_n : 4) : 0;
#define TB_GEMM2_CASE(AM, BMN, O) \
  if (a_mn == AM && b_mn == BMN && out_mode == O) \
    return launch_pairs(gemm2_bf16_kernel<AM, BMN, O>, units, num_sms, stream, ta, tb_, tc, M, N, K, splits, \
                        static_cast<int>(slice_rows), group, err);
  TB_GEMM2_CASE(false, false, 0)
  TB_GEMM2_CASE(false, false, 1)
  TB_GEMM2_CASE(false, false, 2)
  TB_GEMM2_CASE(false, true, 0)
  TB_GEMM2_CASE(false, true, 1)
  TB_GEMM2_CASE(true, true, 0)
  TB_GEMM2_CASE(true, true, 1)
  TB_GEMM2_CASE(true, true, 2)
  TB_GEMM2_CASE(true, false, 0)
#undef TB_GEMM2_CASE
  return -2;
}

int gemm2_swiglu(const void* A, const void* W, void* gu, void* act, int M, int F, int K, int64_t lda, int64_t ldw, int* err,
                 int num_sms, cudaStream_t stream) {
  CUtensorMap ta, tw, tg, tu, tact;
  int r = make_tmap_2d(&ta, A, 2, M, K, lda, BM, 64);
  if (r) return r;
  r = make_tmap_2d(&tw, W, 2, 2 * static_cast<uint64_t>(F), K, ldw, BNH, 64);
  if (r) return r - 100;
  r = make_tmap_2d(&tact, act, 2, M, F, F, 32, 64);
  if (r) return r - 200;
  tg = tu = tact;
  if (gu != nullptr) {
    // one map per half: a store past column F of the gate half must not reach the up half
    r = make_tmap_2d(&tg, gu, 2, M, F, 2 * static_cast<int64_t>(F), 32, 64);
    if (!r) r = make_tmap_2d(&tu, reinterpret_cast<__nv_bfloat16*>(gu) + F, 2, M, F, 2 * static_cast<int64_t>(F), 32, 64);
    if (r) return r - 300;
  }
  EpiArgs ea{};
  ea.store = gu != nullptr ? 1 : 0;
  const int units = ((M + 2 * BM - 1) / (2 * BM)) * ((F + BNH - 1) / BNH);
  return launch_pairs(gemm2_swiglu_kernel, units, num_sms, stream, ta, tw, tg, tu, tact, ea, M, F, K, err);
}

// K of 2048 and more, and tiles for 3.25 waves of SM pairs and more.  Measured on B200, M x F x K (waves): product + pass over it,
// fused, in us.
//   K too short     8192 x 3072 x 512 (5.2) 74.9, 79.8; 8192 x 3072 x 1024 92.5, 93.6; 4096 x 9728 x 512 (8.2) 110.5, 114.1
//   too few waves   2048 x 3072 x 2048 (1.3) 41.3, 45.4; 512 x 9728 x 2560 (1.03) 44.9, 49.3; 1024 x 9728 x 2048 (2.05) 57.9, 60.4;
//                   1408 x 9728 x 2560 (3.08) 85.2, 87.0; 1024 x 14336 x 2048 (3.03) 77.3, 77.5
//   taken           8192 x 2048 x 2048 (3.5) 80.4, 73.8; 6144 x 3072 x 2560 (3.9) 95.5, 92.0; 2048 x 9728 x 2560 (4.1) 106.3,
//                   104.8; 4096 x 9728 x 2560 (8.2) 194, 185; 8192 x 8192 x 2048 (13.8) 273, 251, x 5120 657, 622
// A few that are left out would gain by it: 8192 x 8192 x 1024 (13.8) 194, 178; 8192 x 1024 x 256 (1.7) 29.5, 28.8.
bool gemm2_swiglu_bwd_pays(int M, int F, int K, int num_sms) {
  const int64_t tiles = static_cast<int64_t>((M + 2 * BM - 1) / (2 * BM)) * ((F + BN - 1) / BN);
  const int pairs = g_pair_capacity > 0 && g_pair_capacity < num_sms / 2 ? g_pair_capacity : num_sms / 2;
  return K >= 2048 && tiles * 4 >= static_cast<int64_t>(pairs) * 13;
}

int gemm2_swiglu_bwd(const void* dy, const void* W, const void* gu, void* dgu, int M, int F, int K, int64_t lda, int64_t ldw,
                     int* err, int num_sms, cudaStream_t stream) {
  if (F % 16 != 0 || (reinterpret_cast<uintptr_t>(gu) & 31) != 0) return -6;
  CUtensorMap ta, tw, tg, tu;
  int r = make_tmap_2d(&ta, dy, 2, M, K, lda, BM, 64);
  if (r) return r;
  r = make_tmap_2d(&tw, W, 2, K, F, ldw, 64, 64);
  if (r) return r - 100;
  r = make_tmap_2d(&tg, dgu, 2, M, F, 2 * static_cast<int64_t>(F), 32, 64);
  if (!r) r = make_tmap_2d(&tu, reinterpret_cast<__nv_bfloat16*>(dgu) + F, 2, M, F, 2 * static_cast<int64_t>(F), 32, 64);
  if (r) return r - 200;
  EpiArgs ea{};
  ea.gu = reinterpret_cast<const __nv_bfloat16*>(gu);
  const int units = ((M + 2 * BM - 1) / (2 * BM)) * ((F + BN - 1) / BN);
  return launch_pairs(gemm2_swiglu_bwd_kernel, units, num_sms, stream, ta, tw, tg, tu, ea, M, F, K, err);
}

int gemm2_ce(const void* A, const void* B, int M, int N, int K, int64_t lda, int64_t ldb, const int64_t* labels, float* stats,
             float* target, int* err, int num_sms, cudaStream_t stream) {
  CUtensorMap ta, tb_;
  int r = make_tmap_2d(&ta, A, 2, M, K, lda, BM, 64);
  if (r) return r;
  r = make_tmap_2d(&tb_, B, 2, N, K, ldb, BNH, 64);
  if (r) return r - 100;
  EpiArgs ea{};
  ea.labels = labels;
  ea.stats = reinterpret_cast<float2*>(stats);
  ea.target = target;
  const int units = ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN);
  return launch_pairs(gemm2_ce_kernel, units, num_sms, stream, ta, tb_, ea, M, N, K, err);
}

}  // namespace tb
