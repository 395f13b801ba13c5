// bf16 GEMM for problems with too few output tiles to fill the chip: one 128 x BN tile (BN = 64, 128 or 256) and one
// slice of K per CTA, the S slices of a tile (S = 1, 2, 4 or 8) being the CTAs of one cluster.
//
// What bounds such a problem is the serial chain of k-blocks of one tile, not the tensor cores: a 600 x 512 x 50257
// product has six 256 x 256 tiles, so the pair kernel ran 786 k-blocks one after the other on 12 SMs, and the 128-row
// products of a short prompt kept 4 to 16 SMs busy.  Narrow tiles and K slices put the same work on up to 148 SMs.
// Measured on B200 (cold weights, pair or single-CTA kernel before -> this kernel), bf16: 128 x 1024 x 1024 9.1 -> 5.6 us,
// 128 x 1024 x 3072 21.2 -> 10.4, 1024 x 512 x 512 9.1 -> 4.8, 2048 x 1024 x 4096 25.4 -> 16.2; in slices of K, which gemm_plan
// takes for a head's gradient, 128 x 1024 x 151936 792 -> 75 (8 slices).
//
//   192 threads: warp 0 TMA producer, warp 1 TMEM allocator + MMA issuer, warps 2..5 epilogue (TMEM lanes), as in
//   gemm_sm100.cu.  S > 1: when every CTA of the cluster has finished its MMAs (its operand stages are free then), each
//   writes its fp32 partial tile through distributed shared memory, BN / S columns to every CTA; each CTA then adds its S
//   partials in slice order and writes its columns.  No workspace, no clear, no atomics: the result has the same bits in
//   every run, and a bf16 output is rounded once from the fp32 sum.
//
// Operand majors and output modes are those of gemm_sm100.cu (mode 2 adds into C: the CTA that owns the columns reads and
// writes them, there is no second writer).  Every wait is bounded.
#include "api.h"
#include "common.cuh"

namespace tb {

int make_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols);

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;             // 16 KB
constexpr int NUM_THREADS = 192;
constexpr int BAR_BYTES = 256;

template <int BN>
struct Plan {
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 64 ? 8 : (BN == 128 ? 6 : 4);     // 192 KB
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + BAR_BYTES + 1024;
  static_assert(BM * BN * 4 <= STAGES * STAGE_BYTES, "the partials of one CTA's columns reuse the operand stages");
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
  return out;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// VEC consecutive columns of one output row (16 bytes: 8 bf16 or 4 fp32), `n` of them inside the matrix.
template <int OUT, int VEC>
__device__ __forceinline__ void put(void* C, int64_t at, float (&f)[VEC], int n) {
  if (OUT == 0) {
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(C) + at;
    if (n >= VEC) {
      uint32_t u[VEC / 2];
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) u[i] = pack_bf16x2(f[2 * i], f[2 * i + 1]);
      *reinterpret_cast<uint4*>(p) = make_uint4(u[0], u[1], u[VEC / 2 - 2], u[VEC / 2 - 1]);
    } else {
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (i < n) p[i] = __float2bfloat16(f[i]);
    }
  } else {
    float* p = reinterpret_cast<float*>(C) + at;
    if (n >= VEC) {
      float4 v = make_float4(f[0], f[1], f[2], f[3]);
      if (OUT == 2) {
        const float4 o = *reinterpret_cast<const float4*>(p);
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      *reinterpret_cast<float4*>(p) = v;
    } else {
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (i < n) p[i] = OUT == 2 ? p[i] + f[i] : f[i];
    }
  }
}

template <bool A_MN, bool B_MN, int OUT, int BN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmC, void* C, int64_t ldc, int M, int N, int K, int splits, int early_b,
                  int* err) {
  // early_b: launched while the kernel before still runs, which has not written B.  Set-up and the first B tiles (weights that
  // come from memory when the problem is small) then run under that kernel's tail; A, and with it everything that
  // follows, waits for its end in the producer thread.
  if (!early_b) {
    pdl_wait();
    pdl_launch_dependents();
  }
  using P = Plan<BN>;
  constexpr int STAGES = P::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // identical in every CTA of the cluster: remote addresses are formed from local ones
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * P::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slice = static_cast<int>(blockIdx.x) % splits;     // == rank in the cluster
  const int tile = static_cast<int>(blockIdx.x) / splits;
  const int num_m = (M + BM - 1) / BM;
  const int m0 = (tile % num_m) * BM, n0 = (tile / num_m) * BN;
  // slices of equal length up to one k-block, none empty (splits <= number of k-blocks)
  const int num_kb = (K + BK - 1) / BK;
  const int kb0 = static_cast<int>(static_cast<int64_t>(num_kb) * slice / splits);
  const int kb1 = static_cast<int>(static_cast<int64_t>(num_kb) * (slice + 1) / splits);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (splits == 1) tma_prefetch_desc(&tmC);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      auto load_b = [&](int st, int k0) {
        uint8_t* sB = smem + st * P::STAGE_BYTES + A_BYTES;
        if (!B_MN) {
          tma_load_2d(sB, &tmB, &full[st], k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sB + j * 8192, &tmB, &full[st], n0 + j * 64, k0);
        }
      };
      const int ahead = early_b ? min(kb1, kb0 + STAGES) : kb0;     // k-blocks whose B is on its way
      if (early_b) {
        for (int kb = kb0; kb < ahead; ++kb) {
          mbar_expect_tx(&full[kb - kb0], P::STAGE_BYTES);
          load_b(kb - kb0, kb * BK);
        }
        pdl_wait();
        pdl_launch_dependents();
      }
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, err, kErrProducerEmptyWait)) break;
        uint8_t* sA = smem + stage * P::STAGE_BYTES;
        if (kb >= ahead) mbar_expect_tx(&full[stage], P::STAGE_BYTES);
        const int k0 = kb * BK;
        if (!A_MN) {
          tma_load_2d(sA, &tmA, &full[stage], k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d(sA + j * 8192, &tmA, &full[stage], m0 + j * 64, k0);
        }
        if (kb >= ahead) load_b(stage, k0);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
      constexpr uint32_t a_lbo = A_MN ? 8192u : 16u, b_lbo = B_MN ? 8192u : 16u;
      constexpr uint32_t a_step = A_MN ? (2048u >> 4) : (32u >> 4);
      constexpr uint32_t b_step = B_MN ? (2048u >> 4) : (32u >> 4);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, err, kErrMmaFullWait)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + stage * P::STAGE_BYTES);
        const uint64_t da = make_desc_sw128(a_addr, a_lbo, 1024);
        const uint64_t db = make_desc_sw128(a_addr + A_BYTES, b_lbo, 1024);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_f16_ss(tmem_base, da + static_cast<uint64_t>(k * a_step), db + static_cast<uint64_t>(k * b_step), idesc,
                      (kb != kb0 || k != 0) ? 1u : 0u);
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tfull);
    }
  }
  __syncwarp();
  bool ok = true;
  if (warp >= 2) {
    ok = mbar_wait_warp(tfull, 0, err, kErrEpilogueTmemFullWait);
    tc_fence_after();
  }
  const int q = warp & 3;                 // TMEM lane quarter an epilogue warp may read
  const int row = q * 32 + lane;
  if (splits == 1) {
    // every slab (32 rows x 128 bytes) has a staging buffer of its own in the idle operand stages
    if (warp >= 2 && ok && m0 + q * 32 < M) {
      constexpr int COLS = OUT == 0 ? 64 : 32;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN / COLS; ++c) {
        if (n0 + c * COLS >= N) break;
        uint32_t v[64];
        __syncwarp();      // one lane stored the slab before
        tmem_ld_32x32b_x32(t_row + c * COLS, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        if (OUT == 0) tmem_ld_32x32b_x32(t_row + c * COLS + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tmem_ld_wait();
        uint8_t* buf = smem + (q * (BN / COLS) + c) * 4096;
        uint8_t* rowp = buf + lane * 128;
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
          *reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4)) = pk;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (OUT == 2) tma_reduce_add_2d(&tmC, buf, n0 + c * COLS, m0 + q * 32);
          else tma_store_2d(&tmC, buf, n0 + c * COLS, m0 + q * 32);
          tma_commit_group();
        }
      }
      if (lane == 0) tma_wait_group<0>();
    }
  } else {
    const int cw = BN / splits;              // columns this CTA owns; BN / 8 >= 8
    const int vecs = cw >> 2;                // 16-byte groups of a partial row
    const int swz = (vecs < 8 ? vecs : 8) - 1;
    const int log_cw = 31 - __clz(cw);
    cluster_sync_all();                      // every CTA's MMAs are done: nobody reads its operand stages any more
    if (warp >= 2) {
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      // slot [slice][row][cw] in the CTA that owns the columns; groups XOR-swizzled by the row against bank conflicts
      const uint32_t base = smem_u32(smem) + static_cast<uint32_t>((slice * BM + row) * cw * 4);
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(t_row + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = c + 4 * j;
          const int dst = col >> log_cw, vec = (col & (cw - 1)) >> 2;
          st_cluster_v4(map_to_cta(base + (static_cast<uint32_t>(vec ^ (row & swz)) << 4), dst), v[4 * j], v[4 * j + 1],
                        v[4 * j + 2], v[4 * j + 3]);
        }
      }
    }
    cluster_sync_all();                      // all partials have arrived; no remote access after this point
    const int col0 = n0 + slice * cw;
    constexpr int VEC = OUT == 0 ? 8 : 4, GRP = VEC / 4;    // 16-byte stores
    const int items = vecs / GRP;
    for (int i = threadIdx.x; i < BM * items; i += NUM_THREADS) {
      const int r = i / items, it = i - r * items;
      const int col = col0 + it * VEC;
      if (m0 + r >= M || col >= N) continue;
      float acc[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
      const uint8_t* p = smem + static_cast<size_t>(r) * cw * 4;
      for (int s = 0; s < splits; ++s, p += static_cast<size_t>(BM) * cw * 4) {
#pragma unroll
        for (int h = 0; h < GRP; ++h) {
          const float4 x = *reinterpret_cast<const float4*>(p + (((it * GRP + h) ^ (r & swz)) << 4));
          acc[4 * h] += x.x; acc[4 * h + 1] += x.y; acc[4 * h + 2] += x.z; acc[4 * h + 3] += x.w;
        }
      }
      put<OUT, VEC>(C, static_cast<int64_t>(m0 + r) * ldc + col, acc, N - col);
    }
  }
  if (*reinterpret_cast<volatile int*>(err) != 0) {
    // a wait expired somewhere: give copies and MMAs in flight time to land before TMEM is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

template <bool A_MN, bool B_MN, int OUT, int BN>
int launch_small(const CUtensorMap& ta, const CUtensorMap& tb_, const CUtensorMap& tc, void* C, int64_t ldc, int M, int N,
                 int K, int splits, int* err, cudaStream_t stream, bool b_is_old) {
  auto kern = gemm_small_kernel<A_MN, B_MN, OUT, BN>;
  if (!ensure_dynamic_smem(reinterpret_cast<const void*>(kern), Plan<BN>::SMEM_BYTES)) return -20;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(((M + BM - 1) / BM) * ((N + BN - 1) / BN) * splits);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = Plan<BN>::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, ta, tb_, tc, C, ldc, M, N, K, splits, b_is_old && pdl_enabled() ? 1 : 0, err) ==
                 cudaSuccess
             ? 0
             : -21;
}

}  // namespace

int gemm_small_bf16(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                    bool a_mn, bool b_mn, int out_mode, int tile_n, int splits, int* err, cudaStream_t stream,
                    bool b_is_old) {
  const int num_kb = (K + BK - 1) / BK;
  if (splits < 1 || splits > 8 || (splits & (splits - 1)) || splits > num_kb) return -3;
  CUtensorMap ta, tb_, tc;
  int r = a_mn ? make_tmap_2d(&ta, A, 2, K, M, lda, 64, 64) : make_tmap_2d(&ta, A, 2, M, K, lda, BM, 64);
  if (r) return r;
  r = b_mn ? make_tmap_2d(&tb_, B, 2, K, N, ldb, 64, 64) : make_tmap_2d(&tb_, B, 2, N, K, ldb, tile_n, 64);
  if (r) return r - 100;
  // checks the alignment of C and ldc, which the direct stores of the split form rely on as well
  r = out_mode == 0 ? make_tmap_2d(&tc, C, 2, M, N, ldc, 32, 64) : make_tmap_2d(&tc, C, 4, M, N, ldc, 32, 32);
  if (r) return r - 200;
#define TB_SMALL_BN(AM, BMN, O, W) \
  if (tile_n == W) return launch_small<AM, BMN, O, W>(ta, tb_, tc, C, ldc, M, N, K, splits, err, stream, b_is_old);
#define TB_SMALL_CASE(AM, BMN, O)                    \
  if (a_mn == AM && b_mn == BMN && out_mode == O) {  \
    TB_SMALL_BN(AM, BMN, O, 64)                      \
    TB_SMALL_BN(AM, BMN, O, 128)                     \
    TB_SMALL_BN(AM, BMN, O, 256)                     \
    return -3;                                       \
  }
  TB_SMALL_CASE(false, false, 0)
  TB_SMALL_CASE(false, false, 1)
  TB_SMALL_CASE(false, false, 2)
  TB_SMALL_CASE(false, true, 0)
  TB_SMALL_CASE(false, true, 1)
  TB_SMALL_CASE(true, true, 0)
  TB_SMALL_CASE(true, true, 1)
  TB_SMALL_CASE(true, true, 2)
  TB_SMALL_CASE(true, false, 0)
#undef TB_SMALL_CASE
#undef TB_SMALL_BN
  return -2;
}

}  // namespace tb
