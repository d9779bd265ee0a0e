// bf16 GEMM for problems that give the persistent kernels too few tiles: one 128 x BN tile (BN 64 or
// 128) per CTA, two CTAs per SM, and for a long contraction over few tiles a cluster of 2 or 4 CTAs
// that split K between them.
//
// What bounds it: latency. A 256x256 pair tile leaves most SMs idle at these sizes and then drains
// 256 columns on four warps; here the tile is small, loads start before the tensor memory is
// allocated, and the accumulator goes through shared memory so that global stores are whole rows.
// A split contraction is summed through distributed shared memory in the order of the K ranges: the
// result does not depend on timing, and there is no workspace to allocate or clear.
#include <math.h>

#include "gemm_core.cuh"
#include "host_common.h"

namespace mm {

constexpr int GT_BM = 128;
constexpr int GT_BK = 64;
constexpr int GT_THREADS = 128;

// The loads in flight set the pace of a CTA (a stage takes about 1.2 us to arrive): 192 KB of ring where
// one CTA has an SM to itself (DEEP), 96 KB where two share it.
template <int BN, bool DEEP>
struct GemmTileCfg {
  static constexpr int kStages = (BN == 64 ? 4 : 3) * (DEEP ? 2 : 1);
  static constexpr int kAStage = GT_BM * GT_BK * 2;
  static constexpr int kBStage = BN * GT_BK * 2;
  static constexpr int kRing = kStages * (kAStage + kBStage);
  static constexpr int kSmem = kRing + 256 + 1024;
  // the fp32 tile reuses the ring; rows are padded by 16 bytes so that eight lanes that write four
  // columns of eight rows each touch different banks
  static constexpr int kRowFloats = BN + 4;
  static_assert(GT_BM * kRowFloats * 4 <= kRing, "the staged tile lies in the ring");
};

__device__ __forceinline__ uint32_t gt_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float4 gt_ld_cluster(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// Stores eight consecutive columns of one row (col0 is a multiple of 8).
template <int OUT>
__device__ __forceinline__ void gt_store8(void* C, int64_t ldc, int row, int col0, int N, float4 a, float4 b, bool vec_ok) {
  float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (OUT == OUT_BF16 || OUT == OUT_BF16_ACC) {
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(C) + static_cast<int64_t>(row) * ldc + col0;
    if (vec_ok && col0 + 8 <= N) {
      if (OUT == OUT_BF16_ACC) {
        const uint4 o = *reinterpret_cast<const uint4*>(p);
        const float2 q0 = unpack_bf16(o.x), q1 = unpack_bf16(o.y), q2 = unpack_bf16(o.z), q3 = unpack_bf16(o.w);
        f[0] += q0.x; f[1] += q0.y; f[2] += q1.x; f[3] += q1.y;
        f[4] += q2.x; f[5] += q2.y; f[6] += q3.x; f[7] += q3.y;
      }
      *reinterpret_cast<uint4*>(p) =
          make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col0 + j < N) p[j] = __float2bfloat16(OUT == OUT_BF16_ACC ? f[j] + __bfloat162float(p[j]) : f[j]);
    }
  } else {
    float* p = reinterpret_cast<float*>(C) + static_cast<int64_t>(row) * ldc + col0;
    if (vec_ok && col0 + 8 <= N) {
      float4* p4 = reinterpret_cast<float4*>(p);
      if (OUT == OUT_F32_ACC) {
        const float4 u = p4[0], w = p4[1];
        a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
        b = make_float4(b.x + w.x, b.y + w.y, b.z + w.z, b.w + w.w);
      }
      p4[0] = a;
      p4[1] = b;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col0 + j < N) p[j] = OUT == OUT_F32_ACC ? f[j] + p[j] : f[j];
    }
  }
}

// The CTA's share of one problem: tile `tile`, K range `rank` of `split`.
template <bool A_MN, bool B_MN, int OUT, int BN, bool DEEP>
__device__ __forceinline__ void gemm_tile_body(const CUtensorMap& tmA, const CUtensorMap& tmB, void* C, int64_t ldc, int M, int N,
                                               int K, int tile, int rank, int split, bool vec_ok, int* __restrict__ err) {
  using Cfg = GemmTileCfg<BN, DEEP>;
  constexpr int ST = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  // the CTAs of a cluster read one another's staged tile: align on the shared-window offset
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sA = smem;
  uint8_t* sB = smem + ST * Cfg::kAStage;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kRing);
  uint64_t* empty = full + ST;
  uint64_t* done = empty + ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int num_m = (M + GT_BM - 1) / GT_BM;
  const int m0 = (tile % num_m) * GT_BM, n0 = (tile / num_m) * BN;
  const int num_kb = (K + GT_BK - 1) / GT_BK;
  const int kb0 = static_cast<int>(static_cast<int64_t>(num_kb) * rank / split);
  const int nkb = static_cast<int>(static_cast<int64_t>(num_kb) * (rank + 1) / split) - kb0;   // >= 1: split <= num_kb

  auto load = [&](int i, int st) {
    const int kb = kb0 + i;
    mbar_expect_tx(&full[st], Cfg::kAStage + Cfg::kBStage);
    uint8_t* a_dst = sA + st * Cfg::kAStage;
    uint8_t* b_dst = sB + st * Cfg::kBStage;
    if (!A_MN) {
      tma_load_2d(a_dst, &tmA, &full[st], kb * GT_BK, m0);
    } else {
#pragma unroll
      for (int j = 0; j < GT_BM / 64; ++j) tma_load_2d(a_dst + j * (GT_BK * 128), &tmA, &full[st], m0 + j * 64, kb * GT_BK);
    }
    if (!B_MN) {
      tma_load_2d(b_dst, &tmB, &full[st], kb * GT_BK, n0);
    } else {
#pragma unroll
      for (int j = 0; j < BN / 64; ++j) tma_load_2d(b_dst + j * (GT_BK * 128), &tmB, &full[st], n0 + j * 64, kb * GT_BK);
    }
  };

  if (warp == 0 && elect_one()) {
    for (int i = 0; i < ST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
    for (int i = 0; i < min(ST, nkb); ++i) load(i, i);   // the ring is empty: nothing to wait for
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot;
  bool ok = true;

  if (warp == 0) {
    if (elect_one()) {
      int st = 0;
      uint32_t phase = 0;
      for (int i = ST; i < nkb; ++i) {
        if (!mbar_wait(&empty[st], phase, err, MM_ERR_WAIT_EMPTY)) { ok = false; break; }
        load(i, st);
        if (++st == ST) { st = 0; phase ^= 1; }
      }
      // an expired wait: give copies that are still in flight time to land before the CTA leaves
      if (!ok)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(GT_BM, BN, A_MN, B_MN);
      const uint64_t desc_a = A_MN ? umma_desc_sw128(smem_u32(sA), GT_BK * 128, 1024) : umma_desc_sw128(smem_u32(sA), 16, 1024);
      const uint64_t desc_b = B_MN ? umma_desc_sw128(smem_u32(sB), GT_BK * 128, 1024) : umma_desc_sw128(smem_u32(sB), 16, 1024);
      int st = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(&full[st], phase, err, MM_ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint64_t da = umma_desc_at(desc_a, st * Cfg::kAStage), db = umma_desc_at(desc_b, st * Cfg::kBStage);
#pragma unroll
        for (int k = 0; k < GT_BK / 16; ++k)
          umma_bf16(tmem_d, umma_desc_at(da, k * (A_MN ? 2048 : 32)), umma_desc_at(db, k * (B_MN ? 2048 : 32)), idesc,
                    (i | k) != 0 ? 1u : 0u);
        umma_commit(&empty[st]);
        if (i == nkb - 1) umma_commit(done);
        if (++st == ST) { st = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (OUT == OUT_F32_ACC || OUT == OUT_BF16_ACC) {
    // the old values come from memory while the contraction runs (64 threads, two rows each)
    constexpr int esz = OUT == OUT_F32_ACC ? 4 : 2;
    const int rows = GT_BM / split;
    for (int r = static_cast<int>(threadIdx.x) - 64; r < rows; r += 64) {
      const int row = m0 + rank * rows + r;
      if (row >= M) break;
      const char* p = reinterpret_cast<const char*>(C) + (static_cast<int64_t>(row) * ldc + n0) * esz;
      const int bytes = min(BN, N - n0) * esz;
      for (int o = 0; o < bytes; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
    }
  }

  // every MMA, and with them every load, of this CTA has completed: the ring becomes the staged tile
  if (!mbar_wait(done, 0, err, MM_ERR_WAIT_TMEM_FULL)) ok = false;
  tc_fence_after();
  float* tile_s = reinterpret_cast<float*>(smem);
  if (ok) {
    float* mine = tile_s + (warp * 32 + lane) * Cfg::kRowFloats;
#pragma unroll
    for (int c = 0; c < BN / 32; ++c) {
      uint32_t r[32];
      tmem_ld_32x32(tmem_d + (static_cast<uint32_t>(warp * 32) << 16) + c * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; ++j)
        reinterpret_cast<float4*>(mine + c * 32)[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                                   __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
    }
  }
  constexpr int LPR = BN / 8;         // lanes per row, eight columns each
  constexpr int RPI = 32 / LPR;       // rows per warp and pass
  const int sub = lane / LPR, col = (lane % LPR) * 8;
  if (split == 1) {
    __syncwarp();                     // a warp stores the 32 rows it staged
    if (ok) {
#pragma unroll 4
      for (int r0 = 0; r0 < 32; r0 += RPI) {
        const int r = warp * 32 + r0 + sub;
        const float4* src = reinterpret_cast<const float4*>(tile_s + r * Cfg::kRowFloats + col);
        if (m0 + r < M && n0 + col < N) gt_store8<OUT>(C, ldc, m0 + r, n0 + col, N, src[0], src[1], vec_ok);
      }
    }
  } else {
    // CTA `rank` sums and stores rows [rank, rank + 1) * 128 / split of the tile
    const int good = __syncthreads_and(ok);
    cluster_sync();
    if (good) {
      const int rows = GT_BM / split, wrows = rows / 4;
      for (int r0 = 0; r0 < wrows; r0 += RPI) {
        if (r0 + sub >= wrows) continue;
        const int r = rank * rows + warp * wrows + r0 + sub;
        const uint32_t at = smem_u32(tile_s + r * Cfg::kRowFloats + col);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        for (int s = 0; s < split; ++s) {
          const float4 u = gt_ld_cluster(at, s), w = gt_ld_cluster(at + 16, s);
          a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
          b = make_float4(b.x + w.x, b.y + w.y, b.z + w.z, b.w + w.w);
        }
        if (m0 + r < M && n0 + col < N) gt_store8<OUT>(C, ldc, m0 + r, n0 + col, N, a, b, vec_ok);
      }
    }
    cluster_sync();                // nobody leaves while a partner may still read its tile
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_d, BN);
  }
}

template <bool A_MN, bool B_MN, int OUT, int BN, bool DEEP>
__global__ void __launch_bounds__(GT_THREADS, DEEP ? 1 : 2)
    gemm_tile_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, void* C, int64_t ldc,
                     int M, int N, int K, int split, bool vec_ok, int* __restrict__ err) {
  gemm_tile_body<A_MN, B_MN, OUT, BN, DEEP>(tmA, tmB, C, ldc, M, N, K, static_cast<int>(blockIdx.x) / split,
                                            static_cast<int>(gt_cluster_rank()), split, vec_ok, err);
}

// Both products of a linear layer's backward pass, dX = dY W and dW (+)= dY^T X, in one launch: neither reads
// what the other writes. A launch costs the host 4..5 us, as long as such a product takes, and two of them fill
// more of the chip. Gradients of a d256 model (eight microbatches of 256 tokens, 128 such pairs): 5.36 -> 4.95 ms.
struct LinearBwd {
  __nv_bfloat16* dx;
  void* dw;
  int T, N, K;         // rows, columns of dY, columns of X
  int dx_tiles;        // CTAs of dX; the others work on dW
  bool dx_vec, dw_vec;
};
template <int OUT_DW, int BN_DX, int BN_DW>
__global__ void __launch_bounds__(GT_THREADS, 1)
    gemm_linear_bwd_kernel(const __grid_constant__ CUtensorMap tmDY, const __grid_constant__ CUtensorMap tmW,
                           const __grid_constant__ CUtensorMap tmDYt, const __grid_constant__ CUtensorMap tmX, LinearBwd p,
                           int* __restrict__ err) {
  const int tile = static_cast<int>(blockIdx.x);
  if (tile < p.dx_tiles)
    gemm_tile_body<false, true, OUT_BF16, BN_DX, true>(tmDY, tmW, p.dx, p.K, p.T, p.K, p.N, tile, 0, 1, p.dx_vec, err);
  else
    gemm_tile_body<true, true, OUT_DW, BN_DW, true>(tmDYt, tmX, p.dw, p.K, p.N, p.K, p.T, tile - p.dx_tiles, 0, 1, p.dw_vec, err);
}

template <int OUT_DW, int BN_DX, int BN_DW>
static int launch_linear_bwd(const CUtensorMap (&tm)[4], const LinearBwd& p, int ctas, cudaStream_t stream) {
  DeviceState* ds = device_state();
  if (!ds) return -1;
  auto kern = gemm_linear_bwd_kernel<OUT_DW, BN_DX, BN_DW>;
  constexpr int smem = GemmTileCfg<BN_DX, true>::kSmem > GemmTileCfg<BN_DW, true>::kSmem ? GemmTileCfg<BN_DX, true>::kSmem
                                                                                        : GemmTileCfg<BN_DW, true>::kSmem;
  static bool configured[kMaxDevices] = {};
  int dev = 0;
  MM_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev]) {
    MM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev] = true;
  }
  kern<<<static_cast<unsigned>(ctas), GT_THREADS, smem, stream>>>(tm[0], tm[1], tm[2], tm[3], p, ds->status);
  MM_LAUNCHED(1);
  return 0;
}
template <int OUT_DW>
static int dispatch_linear_bwd(int bn_dx, int bn_dw, const CUtensorMap (&tm)[4], const LinearBwd& p, int ctas, cudaStream_t stream) {
  if (bn_dx == 64) return bn_dw == 64 ? launch_linear_bwd<OUT_DW, 64, 64>(tm, p, ctas, stream) : launch_linear_bwd<OUT_DW, 64, 128>(tm, p, ctas, stream);
  return bn_dw == 64 ? launch_linear_bwd<OUT_DW, 128, 64>(tm, p, ctas, stream) : launch_linear_bwd<OUT_DW, 128, 128>(tm, p, ctas, stream);
}

template <bool A_MN, bool B_MN, int OUT, int BN, bool DEEP>
static int launch_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, void* C, int64_t ldc, int M, int N, int K, int split,
                       bool vec_ok, cudaStream_t stream) {
  DeviceState* ds = device_state();
  if (!ds) return -1;
  auto kern = gemm_tile_kernel<A_MN, B_MN, OUT, BN, DEEP>;
  constexpr int smem = GemmTileCfg<BN, DEEP>::kSmem;
  static bool configured[kMaxDevices] = {};
  int dev = 0;
  MM_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev]) {
    MM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev] = true;
  }
  const int64_t tiles = static_cast<int64_t>((M + GT_BM - 1) / GT_BM) * ((N + BN - 1) / BN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles * split), 1, 1);
  cfg.blockDim = dim3(GT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 1 : 0;
  MM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, C, ldc, M, N, K, split, vec_ok, ds->status));
  count_launches(1);
  return 0;
}

template <bool A_MN, bool B_MN, int BN, bool DEEP>
static int dispatch_mode(int out_mode, const CUtensorMap& tmA, const CUtensorMap& tmB, void* C, int64_t ldc, int M, int N,
                         int K, int split, bool vec_ok, cudaStream_t stream) {
  switch (out_mode) {
    case OUT_BF16: return launch_tile<A_MN, B_MN, OUT_BF16, BN, DEEP>(tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
    case OUT_F32: return launch_tile<A_MN, B_MN, OUT_F32, BN, DEEP>(tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
    case OUT_F32_ACC: return launch_tile<A_MN, B_MN, OUT_F32_ACC, BN, DEEP>(tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
    case OUT_BF16_ACC: return launch_tile<A_MN, B_MN, OUT_BF16_ACC, BN, DEEP>(tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
  }
  return -3;
}

template <bool A_MN, bool B_MN, int BN>
static int dispatch_tile(int out_mode, const CUtensorMap& tmA, const CUtensorMap& tmB, void* C, int64_t ldc, int M, int N,
                         int K, int split, bool vec_ok, cudaStream_t stream) {
  DeviceState* ds = device_state();
  if (!ds) return -1;
  const int64_t ctas = static_cast<int64_t>((M + GT_BM - 1) / GT_BM) * ((N + BN - 1) / BN) * split;
  return ctas <= ds->sm_count ? dispatch_mode<A_MN, B_MN, BN, true>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream)
                              : dispatch_mode<A_MN, B_MN, BN, false>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
}

template <int BN>
static int run_tile(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int out_mode,
                    int64_t ldc, int M, int N, int K, int split, cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc = a_mn ? encode_tmap_2d_bf16(&tmA, A, M, K, lda * 2, 64, GT_BK) : encode_tmap_2d_bf16(&tmA, A, K, M, lda * 2, GT_BK, GT_BM);
  if (rc) return rc;
  rc = b_mn ? encode_tmap_2d_bf16(&tmB, B, N, K, ldb * 2, 64, GT_BK) : encode_tmap_2d_bf16(&tmB, B, K, N, ldb * 2, GT_BK, BN);
  if (rc) return rc;
  const int esz = (out_mode == OUT_BF16 || out_mode == OUT_BF16_ACC) ? 2 : 4;
  const bool vec_ok = ((ldc * esz) % 16 == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
  if (!a_mn && !b_mn) return dispatch_tile<false, false, BN>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
  if (!a_mn && b_mn) return dispatch_tile<false, true, BN>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
  if (a_mn && b_mn) return dispatch_tile<true, true, BN>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
  return dispatch_tile<true, false, BN>(out_mode, tmA, tmB, C, ldc, M, N, K, split, vec_ok, stream);
}

// Kernel and tile of a product: small tiles (`bn`, `split`) where `cols` is 0, else a persistent kernel on `cols` columns.
struct GemmChoice {
  int bn, split, cols;
  bool pair;
};
static GemmChoice gemm_choose(int out_mode, int M, int N, int K, bool b_mn, int64_t lda, int64_t ldb, int pair_min_m, int sm) {
  const double kb = (K + GT_BK - 1) / GT_BK;
  auto blocks = [&](int bm, int bn) { return static_cast<double>((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  auto rounds = [](double ctas, int at_once) { return ceil(ctas / at_once); };
  const bool f32 = out_mode == OUT_F32 || out_mode == OUT_F32_ACC;
  const bool acc = out_mode == OUT_F32_ACC || out_mode == OUT_BF16_ACC;
  const double fresh = 0.035 * (static_cast<double>(M) + N) * (2e-6 * GT_BK);    // us per K block: its operands in MB
  const double part = fmin(1.0, N / 256.0);                                     // of a persistent tile's columns
  auto single_time = [&](int n) {
    return 6.0 + (acc ? 6.0 : f32 ? 2.0 : 0.0) * part * (n / 256.0) + rounds(blocks(128, n), sm) * kb * (0.10 + 0.30 * (n / 256.0) + fresh);
  };
  auto pair_time = [&](int n) {
    const double tiles = blocks(256, n), full = tiles < sm / 2 ? tiles / (sm / 2) : 1.0;
    return 5.3 + (acc ? 4.2 : f32 ? 1.2 : 0.0) * part * (n / 256.0) +
           rounds(tiles, sm / 2) * kb * (0.08 + 0.22 * (n / 256.0) + (0.05 + fresh) * full);
  };
  const bool pairs = pair_min_m > 0 && M >= pair_min_m;
  double best = single_time(256);
  bool pair = false;
  if (pairs && pair_time(256) < best) { best = pair_time(256); pair = true; }
  int bn = 0, split = 0;
  for (int n = 64; n <= 128; n += 64) {
    for (int s = 1; s <= 4 && s <= kb; s *= 2) {
      const double ctas = blocks(128, n) * s, k = ceil(kb / s);
      if (s > 1 && ctas > sm) break;      // a split pays only for SMs that would have stood idle
      double t = (n == 64 ? 3.4 : 4.0) + (acc ? (n == 64 ? 1.5 : 3.0) / s : 0.0) + (s > 1 ? 2.5 + 0.1 * s : 0.0);
      if (ctas <= sm)
        t += k * (n == 64 ? 0.162 : 0.215 + fresh);
      else
        t += rounds(ctas, 2 * sm) * (k * ((n == 64 ? 0.31 : ctas <= 2 * sm ? 0.415 : 0.50) + (ctas <= 2 * sm ? 4.6 : 2.9) * fresh) + 1.0);
      if (t < best) { best = t; bn = n; split = s; }
    }
  }
  // narrower tiles: see mm_gemm_auto_bf16
  int cols = bn ? 0 : 256;      // of a persistent tile
  double narrow = 0.95 * best;
  if (bn || pair) {
    const bool sectors = lda % 16 == 0 && ldb % 16 == 0;
    const bool one_round = bn == 64 && blocks(128, 64) * split <= 2 * sm;
    if (pairs && narrow > 5.3 && (!b_mn || sectors) && !one_round && !(acc && kb < (bn ? 8 : 4)))
      for (int n = 128; n < 256; n += 32)
        if (pair_time(n) < narrow) { narrow = pair_time(n); pair = true; cols = n; }
  } else if (!b_mn && narrow > 6.0) {
    for (int n = 128; n < 256; n += 16)
      if (single_time(n) < narrow) { narrow = single_time(n); cols = n; }
  }
  return GemmChoice{bn, split, cols, pair};
}

}  // namespace mm

extern "C" {

int mm_gemm_cols_bf16(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int out_mode,
                      int64_t ldc, int M, int N, int K, int bn, cudaStream_t stream);
int mm_gemm_pair_cols_bf16(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int out_mode,
                           int64_t ldc, int M, int N, int K, int bn, cudaStream_t stream);

// Same contract as mm_gemm_bf16 on 128 x bn tiles (bn: 64 or 128) with the contraction split over
// `split` CTAs (1, 2 or 4, at most one per 64 elements of K).
int mm_gemm_tile_bf16(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int out_mode,
                      int64_t ldc, int M, int N, int K, int bn, int split, cudaStream_t stream) {
  using namespace mm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8)) {
    fprintf(stderr, "[mm_kernels] gemm: leading dimensions must be multiples of 8 elements\n");
    return -2;
  }
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) {
    fprintf(stderr, "[mm_kernels] gemm: operands must be 16-byte aligned\n");
    return -2;
  }
  if ((split != 1 && split != 2 && split != 4) || split > (K + GT_BK - 1) / GT_BK) return -2;
  if (bn == 64) return run_tile<64>(A, a_mn, lda, B, b_mn, ldb, C, out_mode, ldc, M, N, K, split, stream);
  if (bn == 128) return run_tile<128>(A, a_mn, lda, B, b_mn, ldb, C, out_mode, ldc, M, N, K, split, stream);
  return -2;
}

static int run_choice(const mm::GemmChoice& c, const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C,
                      int out_mode, int64_t ldc, int M, int N, int K, cudaStream_t stream) {
  if (!c.cols) return mm_gemm_tile_bf16(A, a_mn, lda, B, b_mn, ldb, C, out_mode, ldc, M, N, K, c.bn, c.split, stream);
  return c.pair ? mm_gemm_pair_cols_bf16(A, a_mn, lda, B, b_mn, ldb, C, out_mode, ldc, M, N, K, c.cols, stream)
                : mm_gemm_cols_bf16(A, a_mn, lda, B, b_mn, ldb, C, out_mode, ldc, M, N, K, c.cols, stream);
}

// Same contract as mm_gemm_bf16; picks the kernel by an estimate of its time in microseconds. Fitted on one
// B200 to cold operands of 64..8192 rows, 256..28672 columns and K 256..28672, where the choice was within
// 8 % of the best of all kernels; both sides where two of them meet (bf16, us):
//   M    N    K      pair  tile 128  tile 64        M     N    K     pair  tile 128  tile 64
//   256  768  256     6.5      5.1      4.0         1500  3072 1024  12.6     12.9     18.2
//   512  512  1536   12.7      9.4      7.7         1500  1024 3072  20.4     15.2     18.7
//   333  4096 4096   25.8     19.4     24.1         500   6144 4096  27.1     31.8     44.6
//   333 28672 4096   89.8     97.9    123.4 (single CTA, 128x256 tiles: 83.0)
// Forward + backward + accumulation of a d256 model (eight microbatches of 256 tokens): 7.87 -> 7.59 ms; of a
// d1024 step on 500-token sequences 2.33 -> 2.17 ms.
// A K block of 64 takes 0.16 us on a 128x64 tile and 0.22 on 128x128 (both bound by what an SM takes in),
// 0.30 .. 0.35 on a 256x256 pair and 0.40 on 128x256 (bound by the tensor cores); what an SM cannot run at once comes in rounds.
// Every MB of operands that a K block brings in - on long, narrow problems nearly all of what the tiles read - costs
// more, most where two small tiles share an SM. Without that term few columns and a long contraction took the small
// tiles and up to twice the time (us, rule by rows alone | before | with the term):
//   29216  280  9088     221   428   221 (pair)        14416   296  5400      79   126    79 (pair)
//    4128 1072 18920     212   324   212 (pair)        10208   176  7400      60    91    60 (pair)
// Of 1,860 random problems (8..32768 rows and columns, K 8..28672) that the terms were not fitted to, 1.2 % lose more
// than a tenth against the rule by rows (before: 2.9 %), the worst of them 2 us of 8 on a size below one tile;
// of 900 problems of model layers (widths 256..4096, 8..8192 tokens) none, and 2 % change their kernel.
// The persistent kernels take narrower tiles where that evens out the last round of the chip: full tiles of 256 columns
// often fill it one and a half times and cost two rounds. A K block's time falls less than its columns (a tile's rows of A
// are read all the same), so the gain has to be more than a twentieth. us, full | narrow tiles:
//    2600 2048 2048   32.8  27.5 (pair, 160)    2048 12288 4096  137.2 123.7 (pair, 224)     600 4096 2048  22.5 20.5 (pair, 192)
//    1024 2816 1500   26.6  23.1 (fp32 accumulation, pair, 160)   5632 1024 1500  38.9  34.8 (the same, 192)
//     333 28672 4096  94.2  90.1 (single, 208; bound by what L2 gives out)
// Only the columns of the kernel that won on full tiles are narrowed (pairs also take over from small tiles that are more
// than the chip holds at once), and not where the narrow tile reads as much as the full one or where that costs most:
//   MN-major B comes in slabs of 64 columns, so that single tiles of 144 read 192: 612 4096 7416 52.9 -> 68.7 on them
//   rows that do not start on the 32 bytes of a sector (MN-major B, whose tiles start anywhere): 1496 4096 3200, rows of
//     1496, 43.8 -> 49.2; 2743 1024 25128 157 -> 181
//   sums into the result over a few K blocks, where reading the result is most of the time: 5120 1024 128 20.8 -> 23.4
// Of 501 problems whose tile changes (model layers and odd sizes up to 8192 rows) the mean gain is 1.12 and five are slower
// by more than 2 %; of 40 whose tile stays two are, which is how far two runs of one kernel differ.
// pair_min_m: CTA pairs from this many rows on; 0: never.
int mm_gemm_auto_bf16(const void* A, int a_mn, int64_t lda, const void* B, int b_mn, int64_t ldb, void* C, int out_mode,
                      int64_t ldc, int M, int N, int K, int pair_min_m, cudaStream_t stream) {
  using namespace mm;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  DeviceState* ds = device_state();
  if (!ds) return -1;
  return run_choice(gemm_choose(out_mode, M, N, K, b_mn != 0, lda, ldb, pair_min_m, ds->sm_count), A, a_mn, lda, B, b_mn, ldb, C,
                    out_mode, ldc, M, N, K, stream);
}

// dx[T, K] = dy[T, N] w[N, K] (bf16) and dw[N, K] (+)= dy^T x[T, K] (dw_mode: an out_mode of mm_gemm_bf16); everything
// contiguous, neither result in memory that the other product reads or writes. One launch where both products would run
// on small tiles and the chip holds all of them at once, else the two calls.
int mm_linear_bwd_bf16(const void* dy, const void* w, const void* x, void* dx, void* dw, int dw_mode, int T, int N, int K,
                       int pair_min_m, cudaStream_t stream) {
  using namespace mm;
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  DeviceState* ds = device_state();
  if (!ds) return -1;
  const GemmChoice a = gemm_choose(OUT_BF16, T, K, N, true, N, K, pair_min_m, ds->sm_count);
  const GemmChoice b = gemm_choose(dw_mode, N, K, T, true, N, K, pair_min_m, ds->sm_count);
  auto ctas = [](int rows, int cols, int bn) { return static_cast<int64_t>((rows + GT_BM - 1) / GT_BM) * ((cols + bn - 1) / bn); };
  const bool aligned = N % 8 == 0 && K % 8 == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
  if (!aligned || dw_mode == OUT_BF16_ACC || a.cols || b.cols || a.split > 1 || b.split > 1 ||
      ctas(T, K, a.bn) + ctas(N, K, b.bn) > ds->sm_count) {
    const int rc = run_choice(a, dy, 0, N, w, 1, K, dx, OUT_BF16, K, T, K, N, stream);
    return rc ? rc : run_choice(b, dy, 1, N, x, 1, K, dw, dw_mode, K, N, K, T, stream);
  }
  CUtensorMap tm[4];
  int rc = encode_tmap_2d_bf16(&tm[0], dy, N, T, static_cast<uint64_t>(N) * 2, GT_BK, GT_BM);
  if (!rc) rc = encode_tmap_2d_bf16(&tm[1], w, K, N, static_cast<uint64_t>(K) * 2, 64, GT_BK);
  if (!rc) rc = encode_tmap_2d_bf16(&tm[2], dy, N, T, static_cast<uint64_t>(N) * 2, 64, GT_BK);
  if (!rc) rc = encode_tmap_2d_bf16(&tm[3], x, K, T, static_cast<uint64_t>(K) * 2, 64, GT_BK);
  if (rc) return rc;
  LinearBwd p;
  p.dx = static_cast<__nv_bfloat16*>(dx);
  p.dw = dw;
  p.T = T;
  p.N = N;
  p.K = K;
  p.dx_tiles = static_cast<int>(ctas(T, K, a.bn));
  p.dx_vec = (reinterpret_cast<uintptr_t>(dx) & 15) == 0;      // rows of K % 8 == 0 elements are multiples of 16 bytes
  p.dw_vec = (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
  const int n = p.dx_tiles + static_cast<int>(ctas(N, K, b.bn));
  switch (dw_mode) {
    case OUT_BF16: return dispatch_linear_bwd<OUT_BF16>(a.bn, b.bn, tm, p, n, stream);
    case OUT_F32: return dispatch_linear_bwd<OUT_F32>(a.bn, b.bn, tm, p, n, stream);
    case OUT_F32_ACC: return dispatch_linear_bwd<OUT_F32_ACC>(a.bn, b.bn, tm, p, n, stream);
  }
  return -3;
}

}  // extern "C"
