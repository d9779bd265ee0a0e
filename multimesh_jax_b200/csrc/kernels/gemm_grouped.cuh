// bf16 GEMM over groups of rows (the tokens routed to each expert) in one launch, on CTA pairs
// (tcgen05.mma.cta_group::2, 256x256 tile per pair; see gemm_pair_core.cuh for the roles).
//
// The rows of all groups lie in one buffer, every group on a multiple of 64 rows with zero rows up
// to the next multiple; starts and counts are read on the device (`plan`), so the host never learns
// them and one launch covers every expert. Two forms:
//
//   rows  : C[r, :] = A[r, :] * B_e          (r in group e; B_e K-major or MN-major, 3-D tensor map, so
//           that a block that runs over the end of one expert's matrix reads zeros, not the next one)
//   wgrad : C_e = A[group e, :]^T * B[group e, :]   (contraction over the group's rows, zero rows included;
//           an empty group stores zeros)
//
// Bound by the tensor cores for long contractions. The tiles of one expert are walked with the row
// block fastest, so a block of weights is read from memory once and from L2 for the other row blocks.
#pragma once
#include "gemm_pair_core.cuh"

namespace mm {

constexpr int GG_MAX_E = 64;
// int32 plan in device memory
constexpr int GG_START = 0;                    // [64] first row of the group (multiple of 64)
constexpr int GG_COUNT = GG_MAX_E;             // [64] rows that hold data
constexpr int GG_TILE = 2 * GG_MAX_E;          // [65] 256-row tiles of the groups before this one
constexpr int GG_PLAN = 3 * GG_MAX_E + 1;
constexpr int GG_PAD = 64;
constexpr int GG_SMEM_BYTES = G2_SMEM_BYTES + 4 * EPI_WARP_BYTES + GG_PLAN * 4 + 12;

struct GroupedShape {
  int E, M, N, K;        // M: wgrad only; K: rows only
  const int* plan;
};

__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x,
                                                 int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Tile `t` of the whole problem: group, blocks, K range. Tiles are visited in ascending order, so the
// group index only moves forward.
template <bool WGRAD>
struct GroupedTiles {
  const int* plan;       // shared-memory copy
  int E, num_n, num_m, num_kb_rows, e = 0;
  __device__ GroupedTiles(const GroupedShape& s, const int* p)
      : plan(p), E(s.E), num_n((s.N + G2_BN - 1) / G2_BN), num_m((s.M + 2 * G2_BM - 1) / (2 * G2_BM)),
        num_kb_rows((s.K + G2_BK - 1) / G2_BK) {}
  __device__ int total() const { return WGRAD ? E * num_m * num_n : plan[GG_TILE + E] * num_n; }
  __device__ void at(int t, int& m_blk, int& n_blk, int& kb0, int& nkb) {
    if (WGRAD) {
      const int per = num_m * num_n;
      e = t / per;
      gemm_tile_coords(t - e * per, num_m, num_n, m_blk, n_blk);
      kb0 = plan[GG_START + e] / G2_BK;
      nkb = (plan[GG_COUNT + e] + G2_BK - 1) / G2_BK;
    } else {
      while (t >= plan[GG_TILE + e + 1] * num_n) ++e;
      const int first = plan[GG_TILE + e], mt = plan[GG_TILE + e + 1] - first;
      const int local = t - first * num_n;
      m_blk = local % mt;
      n_blk = local / mt;
      kb0 = 0;
      nkb = num_kb_rows;
    }
  }
};

template <bool B_MN, bool WGRAD>
__global__ void __launch_bounds__(G2_THREADS, 1)
    gemm_grouped_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GroupedShape shape,
                        __nv_bfloat16* __restrict__ C, int64_t ldc, int64_t group_stride, bool vec_ok, int* __restrict__ err) {
  constexpr bool A_MN = WGRAD;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sA = smem;
  uint8_t* sB = smem + G2_STAGES * G2_A_STAGE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G2_STAGES * G2_STAGE_BYTES);
  uint64_t* full = bars;                   // [STAGES]  used in the leader only
  uint64_t* empty = bars + G2_STAGES;      // [STAGES]  one set per CTA
  uint64_t* tfull = bars + 2 * G2_STAGES;  // [2]       one set per CTA
  uint64_t* tempty = tfull + 2;            // [2]       used in the leader only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  uint8_t* epi_stage = smem + G2_STAGES * G2_STAGE_BYTES + 256;
  int* plan = reinterpret_cast<int*>(epi_stage + 4 * EPI_WARP_BYTES);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int i = 0; i < G2_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  for (int i = threadIdx.x; i < GG_PLAN; i += blockDim.x) plan[i] = shape.plan[i];
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  GroupedTiles<WGRAD> tiles(shape, plan);
  const int num_tiles = tiles.total();
  int m_blk, n_blk, kb0, nkb;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile, m_blk, n_blk, kb0, nkb);
        const int m0 = (m_blk * 2 + static_cast<int>(rank)) * G2_BM;
        const int a0 = WGRAD ? m0 : plan[GG_START + tiles.e] + m0;
        const int b0 = n_blk * G2_BN + static_cast<int>(rank) * G2_BNH;
        for (int i = 0; i < nkb; ++i) {
          if (!mbar_wait(&empty[stage], phase ^ 1, err, MM_ERR_WAIT_EMPTY)) { ok = false; break; }
          if (leader) mbar_expect_tx(&full[stage], 2 * G2_STAGE_BYTES);
          const uint32_t bar = mapa_u32(&full[stage], 0);
          uint8_t* a_dst = sA + stage * G2_A_STAGE;
          uint8_t* b_dst = sB + stage * G2_B_STAGE;
          const int k0 = (kb0 + i) * G2_BK;
          if (!A_MN) {
            tma_load_2d_pair(a_dst, &tmA, bar, k0, a0);
          } else {
#pragma unroll
            for (int j = 0; j < G2_BM / 64; ++j) tma_load_2d_pair(a_dst + j * (G2_BK * 128), &tmA, bar, a0 + j * 64, k0);
          }
          if (WGRAD) {
#pragma unroll
            for (int j = 0; j < G2_BNH / 64; ++j) tma_load_2d_pair(b_dst + j * (G2_BK * 128), &tmB, bar, b0 + j * 64, k0);
          } else if (B_MN) {
#pragma unroll
            for (int j = 0; j < G2_BNH / 64; ++j)
              tma_load_3d_pair(b_dst + j * (G2_BK * 128), &tmB, bar, b0 + j * 64, k0, tiles.e);
          } else {
            tma_load_3d_pair(b_dst, &tmB, bar, k0, b0, tiles.e);
          }
          if (++stage == G2_STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // give copies that are still in flight time to land before the pair leaves
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      const uint64_t desc_a = A_MN ? umma_desc_sw128(smem_u32(sA), G2_BK * 128, 1024) : umma_desc_sw128(smem_u32(sA), 16, 1024);
      const uint64_t desc_b = (B_MN || WGRAD) ? umma_desc_sw128(smem_u32(sB), G2_BK * 128, 1024) : umma_desc_sw128(smem_u32(sB), 16, 1024);
      constexpr uint32_t idesc = umma_idesc_bf16(2 * G2_BM, G2_BN, A_MN, B_MN || WGRAD);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile, m_blk, n_blk, kb0, nkb);
        if (nkb == 0) continue;      // an empty group: the epilogue stores zeros without an accumulator
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, err, MM_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * G2_BN;
        for (int i = 0; i < nkb; ++i) {
          if (!mbar_wait(&full[stage], phase, err, MM_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint64_t da = umma_desc_at(desc_a, stage * G2_A_STAGE), db = umma_desc_at(desc_b, stage * G2_B_STAGE);
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k)
            umma_bf16_pair(d_tmem, umma_desc_at(da, k * (A_MN ? 2048 : 32)), umma_desc_at(db, k * ((B_MN || WGRAD) ? 2048 : 32)), idesc,
                           (i | k) != 0 ? 1u : 0u);
          umma_commit_pair(&empty[stage], 3);   // frees the stage in both CTAs
          if (++stage == G2_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(&tfull[acc], 3);       // both halves of the accumulator are complete
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      tiles.at(tile, m_blk, n_blk, kb0, nkb);
      const int local = (m_blk * 2 + static_cast<int>(rank)) * G2_BM + q * 32 + lane;
      // rows: the zero rows behind the group's data are stored too (the next contraction reads them)
      const int limit = WGRAD ? shape.M : (plan[GG_COUNT + tiles.e] + GG_PAD - 1) / GG_PAD * GG_PAD;
      __nv_bfloat16* base = WGRAD ? C + tiles.e * group_stride : C + static_cast<int64_t>(plan[GG_START + tiles.e]) * ldc;
      const int ncol = min(G2_BN, shape.N - n_blk * G2_BN);
      if (nkb == 0) {
        uint32_t z[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) z[j] = 0;
        for (int c = 0; c < ncol; c += 32)
          if (local < limit) gemm_store_chunk<OUT_BF16>(base, ldc, local, n_blk * G2_BN + c, shape.N, z, vec_ok);
        continue;
      }
      if (!mbar_wait(&tfull[acc], acc_phase, err, MM_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t t_base = tmem_base + acc * G2_BN + (static_cast<uint32_t>(q * 32) << 16);
      if (vec_ok && ncol % 8 == 0) {
        gemm_drain_warp<OUT_BF16>(t_base, base, ldc, local - lane, limit, n_blk * G2_BN, ncol, epi_stage + q * EPI_WARP_BYTES, lane);
      } else {
#pragma unroll 1
        for (int c = 0; c < ncol; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(t_base + c, r);
          tmem_ld_wait();
          if (local < limit) gemm_store_chunk<OUT_BF16>(base, ldc, local, n_blk * G2_BN + c, shape.N, r, vec_ok);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(&tempty[acc], 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  // nobody leaves, and no TMEM is freed, while the partner may still signal this CTA's barriers
  // or run MMAs on its tensor memory
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Launches at most one pair per two SMs, and no more than `max_tiles`.
template <bool B_MN, bool WGRAD>
static int launch_grouped(const CUtensorMap& tmA, const CUtensorMap& tmB, const GroupedShape& shape, void* C, int64_t ldc,
                          int64_t group_stride, int64_t max_tiles, cudaStream_t stream) {
  DeviceState* ds = device_state();
  if (!ds) return -1;
  auto kern = gemm_grouped_kernel<B_MN, WGRAD>;
  static bool configured[kMaxDevices] = {};
  int dev = 0;
  MM_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev]) {
    MM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GG_SMEM_BYTES));
    configured[dev] = true;
  }
  const int64_t pairs = max_tiles < ds->sm_count / 2 ? max_tiles : ds->sm_count / 2;
  if (pairs < 1) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
  cfg.blockDim = dim3(G2_THREADS, 1, 1);
  cfg.dynamicSmemBytes = GG_SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool vec_ok = (ldc % 8 == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0) && (group_stride % 8 == 0);
  MM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, shape, static_cast<__nv_bfloat16*>(C), ldc, group_stride, vec_ok, ds->status));
  return 0;
}

// C[r, N] = A[r, K] * B_e over the rows of every group. A [rows_cap, K]; B [E, N, K] (b_mn == 0) or
// [E, K, N] (b_mn == 1); everything contiguous.
static int grouped_rows(const void* A, const void* B, int b_mn, void* C, int rows_cap, int E, int N, int K, const int* plan,
                        cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc = encode_tmap_2d_bf16(&tmA, A, K, rows_cap, static_cast<uint64_t>(K) * 2, G2_BK, G2_BM);
  if (rc) return rc;
  const uint64_t inner = b_mn ? N : K, outer = b_mn ? K : N;
  const uint64_t dims[3] = {inner, outer, static_cast<uint64_t>(E)};
  const uint64_t strides[3] = {0, inner * 2, inner * outer * 2};
  const uint32_t box[3] = {64, static_cast<uint32_t>(b_mn ? G2_BK : G2_BNH), 1};
  rc = encode_tmap_bf16(&tmB, B, 3, dims, strides, box, 1);
  if (rc) return rc;
  GroupedShape s{E, 0, N, K, plan};
  const int64_t max_tiles = (static_cast<int64_t>(rows_cap) / (2 * G2_BM) + E) * ((N + G2_BN - 1) / G2_BN);
  return b_mn ? launch_grouped<true, false>(tmA, tmB, s, C, N, 0, max_tiles, stream)
              : launch_grouped<false, false>(tmA, tmB, s, C, N, 0, max_tiles, stream);
}

// C_e[M, N] = A[group e, M]^T * B[group e, N]; C [E, M, N].
static int grouped_wgrad(const void* A, const void* B, void* C, int rows_cap, int E, int M, int N, const int* plan,
                         cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc = encode_tmap_2d_bf16(&tmA, A, M, rows_cap, static_cast<uint64_t>(M) * 2, 64, G2_BK);
  if (rc) return rc;
  rc = encode_tmap_2d_bf16(&tmB, B, N, rows_cap, static_cast<uint64_t>(N) * 2, 64, G2_BK);
  if (rc) return rc;
  GroupedShape s{E, M, N, 0, plan};
  const int64_t tiles = static_cast<int64_t>(E) * ((M + 2 * G2_BM - 1) / (2 * G2_BM)) * ((N + G2_BN - 1) / G2_BN);
  return launch_grouped<true, true>(tmA, tmB, s, C, N, static_cast<int64_t>(M) * N, tiles, stream);
}

}  // namespace mm
