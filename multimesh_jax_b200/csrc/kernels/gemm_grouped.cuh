// bf16 GEMM over groups of rows (the tokens routed to each expert) in one launch, on CTA pairs
// (tcgen05.mma.cta_group::2; see gemm_pair_core.cuh for the roles).
//
// The rows of all groups lie in one buffer, every group on a multiple of 64 rows with zero rows up
// to the next multiple; starts and counts are read on the device (`plan`), so the host never learns
// them and one launch covers every expert. Two forms:
//
//   rows  : C[r, :] = A[r, :] * B_e          (r in group e; B_e K-major or MN-major, 3-D tensor map, so
//           that a block that runs over the end of one expert's matrix reads zeros, not the next one).
//           The pair's 256 accumulator rows are columns of C and the tile's columns are rows of the group:
//           their number is the instruction's N, any multiple of 32, so a group is cut into equal tiles
//           that fit it. With 256 rows of the group per tile an expert with 1,040 rows paid for 1,280. Five such
//           products of a block forward + backward, us, 256 rows | equal tiles (D 4096): 4096 tokens of F 14336
//           6409 | 5950, 1100 of F 8192 1772 | 1148, 257 of F 14336 1458 | 1240; 300 of D 512 F 1024 54 | 48.
//   wgrad : C_e = A[group e, :]^T * B[group e, :]   (contraction over the group's rows, zero rows included;
//           an empty group stores zeros)
//
// Bound by the tensor cores for long contractions. The tiles of one expert are walked with the group's
// rows fastest, so a block of weights is read from memory once and from L2 for the other tiles.
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

// What the two kernels share: barriers, tensor memory, the plan in shared memory.
struct GroupedSmem {
  uint8_t *sA, *sB, *epi;
  uint64_t *full, *empty, *tfull, *tempty;   // full, tempty: used in the leader only; empty, tfull: one set per CTA
  uint32_t* tmem_slot;
  int* plan;
  __device__ GroupedSmem(uint8_t* raw) {
    const uint32_t at = smem_u32(raw);
    uint8_t* smem = raw + (((at + 1023u) & ~1023u) - at);
    sA = smem;
    sB = smem + G2_STAGES * G2_A_STAGE;
    full = reinterpret_cast<uint64_t*>(smem + G2_STAGES * G2_STAGE_BYTES);
    empty = full + G2_STAGES;
    tfull = empty + G2_STAGES;
    tempty = tfull + 2;
    tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    epi = smem + G2_STAGES * G2_STAGE_BYTES + 256;
    plan = reinterpret_cast<int*>(epi + 4 * EPI_WARP_BYTES);
  }
  // Returns the tensor memory's base.
  __device__ uint32_t begin(const CUtensorMap* a, const CUtensorMap* b, const int* plan_dev) {
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
      tma_prefetch_desc(a);
      tma_prefetch_desc(b);
    }
    if (warp_index() == 1) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    }
    for (int i = threadIdx.x; i < GG_PLAN; i += blockDim.x) plan[i] = plan_dev[i];
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    return *tmem_slot;
  }
  // Nobody leaves, and no TMEM is freed, while the partner may still signal this CTA's barriers
  // or run MMAs on its tensor memory.
  __device__ void end(uint32_t tmem_base) {
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp_index() == 1) {
      tc_fence_after();
      tmem_dealloc_pair(tmem_base, 512);
    }
  }
};

// Tile `t` of the rows form: group, block of 256 columns of C, rows of the group. Tiles are visited in ascending
// order, so the group index only moves forward.
struct RowTiles {
  const int* plan;       // shared-memory copy
  int E, num_n, e = 0;
  int n_blk, row0, rows, width, stored;   // row0: of the buffer; rows: of the tile; stored: rows of the group, zero rows included
  __device__ RowTiles(const GroupedShape& s, const int* p) : plan(p), E(s.E), num_n((s.N + 2 * G2_BM - 1) / (2 * G2_BM)) {}
  __device__ int total() const { return plan[GG_TILE + E] * num_n; }
  __device__ void at(int t) {
    while (t >= plan[GG_TILE + e + 1] * num_n) ++e;
    const int first = plan[GG_TILE + e], tiles = plan[GG_TILE + e + 1] - first;
    const int local = t - first * num_n, j = local % tiles;
    n_blk = local / tiles;
    stored = (plan[GG_COUNT + e] + GG_PAD - 1) / GG_PAD * GG_PAD;
    width = ((stored + tiles - 1) / tiles + 31) / 32 * 32;     // <= 256: a group has a tile for every 256 rows
    row0 = plan[GG_START + e] + j * width;
    rows = min(width, stored - j * width);                     // the last tile may be short, or have none
  }
};

template <bool W_MN>
__global__ void __launch_bounds__(G2_THREADS, 1)
    gemm_grouped_rows_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, GroupedShape shape,
                             __nv_bfloat16* __restrict__ C, int64_t ldc, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  GroupedSmem sm(smem_raw);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const uint32_t tmem_base = sm.begin(&tmX, &tmW, shape.plan);
  RowTiles tiles(shape, sm.plan);
  const int num_tiles = tiles.total();
  const int num_kb = (shape.K + G2_BK - 1) / G2_BK;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile);
        const int w0 = tiles.n_blk * (2 * G2_BM) + rank * G2_BM;
        const int x0 = tiles.row0 + rank * (tiles.width / 2);    // the box is 128 rows whatever the width
        for (int i = 0; i < num_kb; ++i) {
          if (!mbar_wait(&sm.empty[stage], phase ^ 1, err, MM_ERR_WAIT_EMPTY)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&sm.full[stage], 2 * G2_STAGE_BYTES);
          const uint32_t bar = mapa_u32(&sm.full[stage], 0);
          uint8_t* w_dst = sm.sA + stage * G2_A_STAGE;
          const int k0 = i * G2_BK;
          if (W_MN) {
#pragma unroll
            for (int j = 0; j < G2_BM / 64; ++j) tma_load_3d_pair(w_dst + j * (G2_BK * 128), &tmW, bar, w0 + j * 64, k0, tiles.e);
          } else {
            tma_load_3d_pair(w_dst, &tmW, bar, k0, w0, tiles.e);
          }
          tma_load_2d_pair(sm.sB + stage * G2_B_STAGE, &tmX, bar, k0, x0);
          if (++stage == G2_STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // give copies that are still in flight time to land before the pair leaves
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const uint64_t desc_w = W_MN ? umma_desc_sw128(smem_u32(sm.sA), G2_BK * 128, 1024) : umma_desc_sw128(smem_u32(sm.sA), 16, 1024);
      const uint64_t desc_x = umma_desc_sw128(smem_u32(sm.sB), 16, 1024);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile);
        const uint32_t idesc = umma_idesc_bf16(2 * G2_BM, tiles.width, W_MN, false);
        if (!mbar_wait(&sm.tempty[acc], acc_phase ^ 1, err, MM_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * G2_BN;
        for (int i = 0; i < num_kb; ++i) {
          if (!mbar_wait(&sm.full[stage], phase, err, MM_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint64_t dw = umma_desc_at(desc_w, stage * G2_A_STAGE), dx = umma_desc_at(desc_x, stage * G2_B_STAGE);
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k)
            umma_bf16_pair(d_tmem, umma_desc_at(dw, k * (W_MN ? 2048 : 32)), umma_desc_at(dx, k * 32), idesc, (i | k) != 0 ? 1u : 0u);
          umma_commit_pair(&sm.empty[stage], 3);   // frees the stage in both CTAs
          if (++stage == G2_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(&sm.tfull[acc], 3);       // both halves of the accumulator are complete
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // A lane holds one column of C over the tile's rows: 32 rows x 32 columns at a time are turned around in shared
    // memory, so that four lanes store 64 consecutive bytes of a row. Two rows of a column go as one word: by single
    // elements the tiles of a short contraction waited for the turn (8000 tokens of D 512 F 1024, gate and up 36.1 ->
    // 34.6 us; with the group's rows on the accumulator's rows, where nothing is turned, 34.7).
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    uint8_t* stage = sm.epi + q * EPI_WARP_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      tiles.at(tile);
      const int col0 = tiles.n_blk * (2 * G2_BM) + rank * G2_BM + q * 32 + (lane & 3) * 8;
      __nv_bfloat16* out = C + static_cast<int64_t>(tiles.row0) * ldc + col0;
      if (!mbar_wait(&sm.tfull[acc], acc_phase, err, MM_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t t_base = tmem_base + acc * G2_BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < tiles.rows; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(t_base + c, v);
        tmem_ld_wait();
        __syncwarp();                            // the previous step's reads are done
        // word = rows 2t, 2t + 1 of a column; neighbouring 16 bytes change places in every other line, so that the eight
        // lanes of a read, which hold two lines, fall into different banks
#pragma unroll
        for (int t = 0; t < 16; ++t)
          reinterpret_cast<uint32_t*>(stage)[t * 32 + (lane ^ ((t & 1) * 4))] = pack_bf16(__uint_as_float(v[2 * t]), __uint_as_float(v[2 * t + 1]));
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = i * 8 + (lane >> 2), k = (lane & 3) * 2;
          const uint4* src = reinterpret_cast<const uint4*>(stage) + t * 8;
          const uint4 a = src[k ^ (t & 1)], b = src[(k + 1) ^ (t & 1)];
          __nv_bfloat16* dst = out + static_cast<int64_t>(c + 2 * t) * ldc;
          if (c + 2 * t < tiles.rows && col0 < shape.N) {      // rows of a tile are a multiple of 32
            *reinterpret_cast<uint4*>(dst) = make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410),
                                                        __byte_perm(b.x, b.y, 0x5410), __byte_perm(b.z, b.w, 0x5410));
            *reinterpret_cast<uint4*>(dst + ldc) = make_uint4(__byte_perm(a.x, a.y, 0x7632), __byte_perm(a.z, a.w, 0x7632),
                                                              __byte_perm(b.x, b.y, 0x7632), __byte_perm(b.z, b.w, 0x7632));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(&sm.tempty[acc], 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }
  sm.end(tmem_base);
}

// Tile `t` of the weight gradients: group, blocks, K range.
struct WgradTiles {
  const int* plan;       // shared-memory copy
  int E, num_n, num_m, e = 0;
  __device__ WgradTiles(const GroupedShape& s, const int* p)
      : plan(p), E(s.E), num_n((s.N + G2_BN - 1) / G2_BN), num_m((s.M + 2 * G2_BM - 1) / (2 * G2_BM)) {}
  __device__ int total() const { return E * num_m * num_n; }
  __device__ void at(int t, int& m_blk, int& n_blk, int& kb0, int& nkb) {
    const int per = num_m * num_n;
    e = t / per;
    gemm_tile_coords(t - e * per, num_m, num_n, m_blk, n_blk);
    kb0 = plan[GG_START + e] / G2_BK;
    nkb = (plan[GG_COUNT + e] + G2_BK - 1) / G2_BK;
  }
};

__global__ void __launch_bounds__(G2_THREADS, 1)
    gemm_grouped_wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GroupedShape shape,
                        __nv_bfloat16* __restrict__ C, int64_t ldc, int64_t group_stride, bool vec_ok, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  GroupedSmem sm(smem_raw);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const uint32_t tmem_base = sm.begin(&tmA, &tmB, shape.plan);
  WgradTiles tiles(shape, sm.plan);
  const int num_tiles = tiles.total();
  int m_blk, n_blk, kb0, nkb;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile, m_blk, n_blk, kb0, nkb);
        const int m0 = (m_blk * 2 + rank) * G2_BM;
        const int b0 = n_blk * G2_BN + rank * G2_BNH;
        for (int i = 0; i < nkb; ++i) {
          if (!mbar_wait(&sm.empty[stage], phase ^ 1, err, MM_ERR_WAIT_EMPTY)) { ok = false; break; }
          if (leader) mbar_expect_tx(&sm.full[stage], 2 * G2_STAGE_BYTES);
          const uint32_t bar = mapa_u32(&sm.full[stage], 0);
          uint8_t* a_dst = sm.sA + stage * G2_A_STAGE;
          uint8_t* b_dst = sm.sB + stage * G2_B_STAGE;
          const int k0 = (kb0 + i) * G2_BK;
#pragma unroll
          for (int j = 0; j < G2_BM / 64; ++j) tma_load_2d_pair(a_dst + j * (G2_BK * 128), &tmA, bar, m0 + j * 64, k0);
#pragma unroll
          for (int j = 0; j < G2_BNH / 64; ++j) tma_load_2d_pair(b_dst + j * (G2_BK * 128), &tmB, bar, b0 + j * 64, k0);
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
      const uint64_t desc_a = umma_desc_sw128(smem_u32(sm.sA), G2_BK * 128, 1024);
      const uint64_t desc_b = umma_desc_sw128(smem_u32(sm.sB), G2_BK * 128, 1024);
      constexpr uint32_t idesc = umma_idesc_bf16(2 * G2_BM, G2_BN, true, true);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        tiles.at(tile, m_blk, n_blk, kb0, nkb);
        if (nkb == 0) continue;      // an empty group: the epilogue stores zeros without an accumulator
        if (!mbar_wait(&sm.tempty[acc], acc_phase ^ 1, err, MM_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * G2_BN;
        for (int i = 0; i < nkb; ++i) {
          if (!mbar_wait(&sm.full[stage], phase, err, MM_ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint64_t da = umma_desc_at(desc_a, stage * G2_A_STAGE), db = umma_desc_at(desc_b, stage * G2_B_STAGE);
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k)
            umma_bf16_pair(d_tmem, umma_desc_at(da, k * 2048), umma_desc_at(db, k * 2048), idesc, (i | k) != 0 ? 1u : 0u);
          umma_commit_pair(&sm.empty[stage], 3);   // frees the stage in both CTAs
          if (++stage == G2_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(&sm.tfull[acc], 3);       // both halves of the accumulator are complete
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
      const int local = (m_blk * 2 + rank) * G2_BM + q * 32 + lane;
      const int limit = shape.M;
      __nv_bfloat16* base = C + tiles.e * group_stride;
      const int ncol = min(G2_BN, shape.N - n_blk * G2_BN);
      if (nkb == 0) {
        uint32_t z[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) z[j] = 0;
        for (int c = 0; c < ncol; c += 32)
          if (local < limit) gemm_store_chunk<OUT_BF16>(base, ldc, local, n_blk * G2_BN + c, shape.N, z, vec_ok);
        continue;
      }
      if (!mbar_wait(&sm.tfull[acc], acc_phase, err, MM_ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t t_base = tmem_base + acc * G2_BN + (static_cast<uint32_t>(q * 32) << 16);
      if (vec_ok && ncol % 8 == 0) {
        gemm_drain_warp<OUT_BF16>(t_base, base, ldc, local - lane, limit, n_blk * G2_BN, ncol, sm.epi + q * EPI_WARP_BYTES, lane);
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
      if (lane == 0) mbar_arrive_cluster(mapa_u32(&sm.tempty[acc], 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  sm.end(tmem_base);
}

// Launches at most one pair per two SMs, and no more than `max_tiles`.
template <class Kernel, class... Args>
static int launch_grouped(Kernel kern, bool (&configured)[kMaxDevices], int64_t max_tiles, cudaStream_t stream, Args... args) {
  DeviceState* ds = device_state();
  if (!ds) return -1;
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
  MM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args..., ds->status));
  count_launches(1);
  return 0;
}

// C[r, N] = A[r, K] * B_e over the rows of every group, the zero rows behind its data included (the next contraction
// reads them). A [rows_cap, K]; B [E, N, K] (b_mn == 0) or [E, K, N] (b_mn == 1); everything contiguous, N a multiple of 8
// and C 16-byte aligned.
static int grouped_rows(const void* A, const void* B, int b_mn, void* C, int rows_cap, int E, int N, int K, const int* plan,
                        cudaStream_t stream) {
  if (N % 8 || (reinterpret_cast<uintptr_t>(C) & 15)) return -2;
  CUtensorMap tmX, tmW;
  int rc = encode_tmap_2d_bf16(&tmX, A, K, rows_cap, static_cast<uint64_t>(K) * 2, G2_BK, G2_BNH);
  if (rc) return rc;
  const uint64_t inner = b_mn ? N : K, outer = b_mn ? K : N;
  const uint64_t dims[3] = {inner, outer, static_cast<uint64_t>(E)};
  const uint64_t strides[3] = {0, inner * 2, inner * outer * 2};
  const uint32_t box[3] = {64, static_cast<uint32_t>(b_mn ? G2_BK : G2_BM), 1};
  rc = encode_tmap_bf16(&tmW, B, 3, dims, strides, box, 1);
  if (rc) return rc;
  const GroupedShape s{E, 0, N, K, plan};
  const int64_t max_tiles = (static_cast<int64_t>(rows_cap) / 256 + E) * ((N + 2 * G2_BM - 1) / (2 * G2_BM));
  static bool configured[2][kMaxDevices] = {};
  auto* c = static_cast<__nv_bfloat16*>(C);
  return b_mn ? launch_grouped(gemm_grouped_rows_kernel<true>, configured[1], max_tiles, stream, tmX, tmW, s, c, static_cast<int64_t>(N))
              : launch_grouped(gemm_grouped_rows_kernel<false>, configured[0], max_tiles, stream, tmX, tmW, s, c, static_cast<int64_t>(N));
}

// C_e[M, N] = A[group e, M]^T * B[group e, N]; C [E, M, N].
static int grouped_wgrad(const void* A, const void* B, void* C, int rows_cap, int E, int M, int N, const int* plan,
                         cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc = encode_tmap_2d_bf16(&tmA, A, M, rows_cap, static_cast<uint64_t>(M) * 2, 64, G2_BK);
  if (rc) return rc;
  rc = encode_tmap_2d_bf16(&tmB, B, N, rows_cap, static_cast<uint64_t>(N) * 2, 64, G2_BK);
  if (rc) return rc;
  const GroupedShape s{E, M, N, 0, plan};
  const int64_t tiles = static_cast<int64_t>(E) * ((M + 2 * G2_BM - 1) / (2 * G2_BM)) * ((N + G2_BN - 1) / G2_BN);
  const int64_t stride = static_cast<int64_t>(M) * N;
  const bool vec_ok = N % 8 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && stride % 8 == 0;
  static bool configured[kMaxDevices] = {};
  return launch_grouped(gemm_grouped_wgrad_kernel, configured, tiles, stream, tmA, tmB, s, static_cast<__nv_bfloat16*>(C),
                        static_cast<int64_t>(N), stride, vec_ok);
}

}  // namespace mm
