// Causal flash attention for sm_100a (head dimension 128, bf16, GQA), forward and backward.
//
// Inputs live in one packed projection buffer [B, S, Hp, 128] with Hp = Hkv * (rep + 2) heads in
// group-major order (per KV head: its `rep` query heads, then the key head, then the value head),
// so query, key and value tiles are all fetched with the same 4-D TMA tensor map. Every matrix
// product runs on the tensor cores through tcgen05.mma with fp32 accumulators in TMEM:
//
//   forward  (128 query rows per CTA, 64 keys per step, two CTAs per SM so that one CTA's softmax
//             overlaps the other's MMAs):
//        S = Q K^T  -> TMEM (double buffered);  softmax threads (one per query row) read S,
//        keep a running maximum that is only raised when it grows by more than 2^8 (the
//        accumulator is then rescaled in TMEM), write P (bf16) over the scores in TMEM, which is where
//        O += P V takes its A operand from; O accumulates in TMEM; epilogue divides by the row sum.
//   backward (128 keys per CTA, 128 query rows per step, every query head of the KV group or a share of them):
//        S^T = K Q^T, dP^T = V dO^T -> TMEM; threads (half a key row each) write P^T (bf16) over the scores, the A
//        operand of dV += P^T dO, and dS^T to shared memory for dK += dS^T Q and dQ = dS K; dV and dK accumulate in
//        TMEM over the whole loop; dQ goes over dP^T's columns and is added to an fp32 buffer by bulk reductions.
//
// Warp roles: forward, warp 0 = TMA producer, warp 1 = MMA issuer and TMEM owner, four softmax / epilogue warps (TMEM
// lane quarter = warp % 4); backward, four warpgroups: TMA and MMA, two of compute warps (two warps per lane quarter,
// splitting the columns) and one that moves dQ, with the registers dealt out anew between them. The backward TMA warp also
// brings the step's log-sum-exp and delta rows into shared memory with the step's Q tile. All waits are bounded.
//
// Ragged sequences run on the same tiles: TMA zero-fills what lies behind the sequence, causality
// masks it for every row inside, and rows outside are not stored. B4 H16 S1000 forward + backward
// takes 0.185 ms against 0.460 ms through the library kernels this replaced. The backward pass has
// one kernel ahead of it (row statistics and the zeroed dQ accumulator) and one behind it (dQ to
// bf16), neither of them for a sequence of one block; both gradients that passed through the rotary
// embedding are rotated back where they are stored, which saves a read-modify-write pass (B1 S8192 32 / 8 heads, whole call: 3.138 -> 3.088 ms).
//
// What the structure rests on, each measured against the other form at the time (ms; the call is forward +
// backward unless it says otherwise):
//   elected issue with ready descriptors (ptx.cuh)      B1 S8192 32 / 8 heads  3.04 -> 2.85, B4 H16 S1000 0.249 -> 0.233
//   forward: exponentials ahead of the wait for the previous product, maximum and sum as four chains each, the
//     scale inside the exponent's multiply-add          B1 S8192 32 / 8 heads  2.83 -> 2.77
//   forward: P through TMEM, not shared memory: at 128 bytes a cycle a step's shared-memory traffic is 1,024 cycles
//     (reads of S 384 and P V 256, K and V tiles 256, P 128), of which 256 go, against 512 of the tensor cores
//                                                       B1 S8192 32 / 8 heads  0.502 -> 0.460, B4 S2048 32 heads 0.171 -> 0.160
//   backward: steps of 128 query rows (N = 64 instructions take as long as N = 128), P^T as an operand in TMEM, dQ by
//     bulk reductions, a KV group's query heads over a cluster where a block would outlast the rest
//       backward  B1 S8192 32 / 8 heads  1.60 -> 1.31   B4 S2048 32 heads  0.643 -> 0.508   B4 S1000 16 heads  0.134 -> 0.112
//                 B3 S500 8 / 2 heads    0.080 -> 0.045  B1 S1500 6 / 2 heads 0.139 -> 0.106  B2 S128 2 heads    0.031 -> 0.025
//     dK and dV in one kernel and dQ in another (seven products instead of five, no sums in memory): 1.52 ms and
//     0.595 ms on the two largest; better only below a dozen blocks
// What bounds it, by counters of B1 S8192 32 / 8 heads: no unit alone. Backward: a step of 128 x 128 is 4,200 cycles, the
// tensor pipe active in 58 % of them; loads and stores of shared memory take 45 % (a third of it bank conflicts), its
// banks are read at 33 % and written at 15 % of their peak, memory is at 10 %. One block per SM has one chain in flight:
// scores, probabilities, dP, dS, dQ, whose columns the next dP waits for. Forward, two blocks per SM: tensor pipe 60 %,
// banks 30 and 16 %, memory 4 %; beside it the exponentials, one per score on the special-function unit.
#include <math.h>

#include <algorithm>

#include "host_common.h"
#include "ptx.cuh"

namespace mm {

constexpr int FA_D = 128;
constexpr int FA_THREADS = 192;
constexpr int MM_ERR_ATTN_WAIT = 7;    // an attention kernel gave up waiting on one of its barriers
constexpr int MM_ERR_ATTN_ALIGN = 8;   // dynamic shared memory was not 1024-byte aligned

// 2^x on the special-function unit alone (ex2.approx.ftz: relative error 2^-22, -inf -> 0): the
// library exp2f adds range scaling around the same instruction, which matters in loops whose
// length is set by the instruction count of one warp (forward: 0.251 -> 0.235 ms on B4 H32 S2048).
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Order in which the blocks of a causal call start. A block's time grows with its distance from the short
// end and the call ends with the last block, so the longest blocks of all heads should start first; but heads
// whose tiles do not fit L2 together are then each read from memory once per block. So heads go in groups,
// and within a group the longest blocks of all its heads start first. A group is what fits a part of L2, or,
// where that is less, as many heads as keep the chip busy for the time of the longest block (twice the
// resident blocks / (blocks of a head + 1)): with fewer the last group ends on a few long blocks.
// Measured, us, head by head | groups by L2 alone | all heads at once | this rule:
//   forward   B1 S8192 32 / 8 heads  554  494  494  502      B4 S2048 32 heads  180  171  174  171
//             B8 S2048  8 heads      104   96   91   92      B4 S1000 16 heads   45   38   40   38
//   backward  B1 S8192 32 / 8 heads 1900 1908 1590 1621      B4 S2048 32 heads  661  646  685  643
//             B8 S2048  8 heads      355  336  330  334      B1 S1024 32 heads   89   73   72   73
struct BlockOrder {
  int heads, group, nblk;   // heads in all, heads of a group, blocks of a head
  // `rank`: 0 for the longest block of its head
  __device__ __forceinline__ void at(int t, int& head, int& rank) const {
    if (nblk == 1) {      // every head one block: a short call feels two divisions
      head = t;
      rank = 0;
      return;
    }
    const int gi = t < group * nblk ? 0 : t / (group * nblk);
    const int within = t - gi * (group * nblk);
    const int n = min(group, heads - gi * group);
    rank = within / n;
    head = gi * group + within - rank * n;
  }
};
constexpr int64_t FA_L2_GROUP_BYTES = 48ll << 20;
// `resident`: blocks that the device runs at once
static BlockOrder block_order(int64_t heads, int64_t bytes_per_head, int nblk, int resident) {
  const int64_t fit = FA_L2_GROUP_BYTES / bytes_per_head, busy = (2 * resident + nblk) / (nblk + 1);
  const int64_t least = fit > busy ? fit : busy;
  const int64_t groups = heads > least ? heads / least : 1;
  return BlockOrder{static_cast<int>(heads), static_cast<int>((heads + groups - 1) / groups), nblk};
}

// ------------------------------------------------------------------ forward
constexpr int FA_BM = 128;
constexpr int FA_BN = 64;
constexpr int FA_SQ = 2 * FA_BM * 128;  // two 64-column halves of 128 rows x 128 B
constexpr int FA_SKV = 2 * FA_BN * 128; // per stage
constexpr int FA_FWD_SMEM = FA_SQ + 4 * FA_SKV + 128;

struct FaFwdParams {
  __nv_bfloat16* out;  // [B, S, Hq, 128]
  float* lse;          // [B, Hq, S]
  int S, Hkv, rep;
  float scale_log2;    // softmax scale * log2(e)
  BlockOrder order;
};

__global__ void __launch_bounds__(FA_THREADS, 2)
    flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                     FaFwdParams p, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) atomicCAS(err, 0, MM_ERR_ATTN_ALIGN);
    return;
  }
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + FA_SQ;
  uint8_t* sV = sK + 2 * FA_SKV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * FA_SKV);
  uint64_t* q_full = bars;          // [1]
  uint64_t* k_full = bars + 1;      // [2]
  uint64_t* k_empty = bars + 3;     // [2]
  uint64_t* v_full = bars + 5;      // [2]
  uint64_t* v_empty = bars + 7;     // [2]
  uint64_t* s_full = bars + 9;      // [2]
  uint64_t* p_ready = bars + 11;    // [1]
  uint64_t* pv_done = bars + 12;    // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  int head, rank;
  p.order.at(blockIdx.x, head, rank);
  const int q_blk = p.order.nblk - 1 - rank;
  const int b = head / (p.Hkv * p.rep), hq = head - b * (p.Hkv * p.rep);
  const int g = hq / p.rep, r = hq - g * p.rep;
  const int hp_q = g * (p.rep + 2) + r, hp_k = g * (p.rep + 2) + p.rep, hp_v = hp_k + 1;
  // key blocks up to the diagonal; a ragged last query block ends with the sequence
  const int nblk = min(2 * q_blk + 2, (p.S + FA_BN - 1) / FA_BN);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(p_ready, 4);
    mbar_init(pv_done, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base;        // two 64-column score buffers; P takes the first 32 columns of its scores
  const uint32_t tO = tmem_base + 128;  // 128-column output accumulator

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, FA_SQ);
      tma_load_4d(sQ, &tmQ, q_full, 0, hp_q, q_blk * FA_BM, b);
      tma_load_4d(sQ + FA_BM * 128, &tmQ, q_full, 64, hp_q, q_blk * FA_BM, b);
      bool ok = true;
      for (int j = 0; j < nblk && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait(&k_empty[st], ph ^ 1, err, MM_ERR_ATTN_WAIT)) { ok = false; break; }
        mbar_expect_tx(&k_full[st], FA_SKV);
        tma_load_4d(sK + st * FA_SKV, &tmKV, &k_full[st], 0, hp_k, j * FA_BN, b);
        tma_load_4d(sK + st * FA_SKV + FA_BN * 128, &tmKV, &k_full[st], 64, hp_k, j * FA_BN, b);
        if (!mbar_wait(&v_empty[st], ph ^ 1, err, MM_ERR_ATTN_WAIT)) { ok = false; break; }
        mbar_expect_tx(&v_full[st], FA_SKV);
        tma_load_4d(sV + st * FA_SKV, &tmKV, &v_full[st], 0, hp_v, j * FA_BN, b);
        tma_load_4d(sV + st * FA_SKV + FA_BN * 128, &tmKV, &v_full[st], 64, hp_v, j * FA_BN, b);
      }
      if (!ok)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies in flight land before exit
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(FA_BM, FA_BN, false, false);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(FA_BM, FA_D, false, true);
      const uint64_t desc_q = umma_desc_sw128(smem_u32(sQ), 16, 1024), desc_k = umma_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t desc_v = umma_desc_sw128(smem_u32(sV), FA_BN * 128, 1024);
      auto issue_s = [&](int j) {
        const int st = j & 1;
        const uint64_t dk = umma_desc_at(desc_k, st * FA_SKV);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_bf16(tS + st * FA_BN, umma_desc_at(desc_q, h * (FA_BM * 128) + kk * 32),
                      umma_desc_at(dk, h * (FA_BN * 128) + kk * 32), idesc_s, (h | kk) ? 1u : 0u);
        umma_commit(&s_full[st]);
        umma_commit(&k_empty[st]);
      };
      bool ok = mbar_wait(q_full, 0, err, MM_ERR_ATTN_WAIT) && mbar_wait(&k_full[0], 0, err, MM_ERR_ATTN_WAIT);
      if (ok) {
        tc_fence_after();
        issue_s(0);
      }
      for (int j = 0; j < nblk && ok; ++j) {
        if (j + 1 < nblk) {
          const int n = j + 1;
          if (!mbar_wait(&k_full[n & 1], (n >> 1) & 1, err, MM_ERR_ATTN_WAIT) ||
              (j > 0 && !mbar_wait(pv_done, (j - 1) & 1, err, MM_ERR_ATTN_WAIT))) { ok = false; break; }   // P of step j - 1 is read
          tc_fence_after();
          issue_s(n);
        }
        if (!mbar_wait(&v_full[j & 1], (j >> 1) & 1, err, MM_ERR_ATTN_WAIT) ||
            !mbar_wait(p_ready, j & 1, err, MM_ERR_ATTN_WAIT)) { ok = false; break; }
        tc_fence_after();
        const uint64_t dv = umma_desc_at(desc_v, (j & 1) * FA_SKV);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts(tO, tS + (j & 1) * FA_BN + kk * 8, umma_desc_at(dv, kk * 2048), idesc_pv, (j | kk) ? 1u : 0u);
        umma_commit(pv_done);
        umma_commit(&v_empty[j & 1]);
      }
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int rowg = q_blk * FA_BM + row;
    const uint32_t lane_bits = static_cast<uint32_t>(q * 32) << 16;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nblk; ++j) {
      const int sb = j & 1;
      if (ok && !mbar_wait(&s_full[sb], (j >> 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
      tc_fence_after();
      uint32_t s0[32], s1[32];
      tmem_ld_32x32(tS + lane_bits + sb * FA_BN, s0);
      tmem_ld_32x32(tS + lane_bits + sb * FA_BN + 32, s1);
      tmem_ld_wait();
      const bool diag = j >= 2 * q_blk;  // the last two key blocks cross the diagonal
      if (diag) {
        const int col0 = j * FA_BN;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (col0 + c > rowg) s0[c] = __float_as_uint(-INFINITY);
          if (col0 + 32 + c > rowg) s1[c] = __float_as_uint(-INFINITY);
        }
      }
      // four independent chains for the maximum and for the sum: one serial chain over the 64 scores
      // took as long as the products of the step
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 32; ++c)
        mx4[c & 3] = fmaxf(mx4[c & 3], fmaxf(__uint_as_float(s0[c]), __uint_as_float(s1[c])));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
      const float m_new = fmaxf(m_used, mx);
      const bool need = m_new > m_used + 8.f;  // raise the reference maximum only on large growth
      float alpha = 1.f;
      if (need) {
        alpha = fast_exp2(m_used - m_new);
        m_used = m_new;
      }
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int c0 = 2 * c, c1 = c0 + 1;
        const float e0 = fast_exp2(fmaf(__uint_as_float(c0 < 32 ? s0[c0 & 31] : s1[c0 & 31]), p.scale_log2, -m_used));
        const float e1 = fast_exp2(fmaf(__uint_as_float(c1 < 32 ? s0[c1 & 31] : s1[c1 & 31]), p.scale_log2, -m_used));
        sum4[c0 & 3] += e0;
        sum4[c1 & 3] += e1;
        pk[c] = pack_bf16(e0, e1);
      }
      l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      // the previous product is still running up to here; it reads P and adds to O
      if (j > 0) {
        if (ok && !mbar_wait(pv_done, (j - 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
        tc_fence_after();
        if (__any_sync(0xffffffffu, need)) {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tO + lane_bits + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(tO + lane_bits + c * 32, o);
          }
          tmem_st_wait();
        }
      }
      tmem_st_32x32(tS + lane_bits + sb * FA_BN, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
    }
    if (ok && !mbar_wait(pv_done, (nblk - 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
    tc_fence_after();
    if (rowg >= p.S) ok = false;   // rows behind the sequence were computed on zero-filled queries
    const float inv = 1.f / l;
    __nv_bfloat16* orow = p.out + ((static_cast<int64_t>(b) * p.S + rowg) * (p.Hkv * p.rep) + hq) * FA_D;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t o[32];
      tmem_ld_32x32(tO + lane_bits + c * 32, o);
      tmem_ld_wait();
      if (ok) {
        uint4* dst = reinterpret_cast<uint4*>(orow + c * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(o[i * 8 + 0]) * inv, __uint_as_float(o[i * 8 + 1]) * inv);
          v.y = pack_bf16(__uint_as_float(o[i * 8 + 2]) * inv, __uint_as_float(o[i * 8 + 3]) * inv);
          v.z = pack_bf16(__uint_as_float(o[i * 8 + 4]) * inv, __uint_as_float(o[i * 8 + 5]) * inv);
          v.w = pack_bf16(__uint_as_float(o[i * 8 + 6]) * inv, __uint_as_float(o[i * 8 + 7]) * inv);
          dst[i] = v;
        }
      }
    }
    if (ok) p.lse[(static_cast<int64_t>(b) * (p.Hkv * p.rep) + hq) * p.S + rowg] = m_used * 0.6931471805599453f + logf(l);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// ------------------------------------------------------------------ backward
constexpr int FB_BLK = 128;               // keys of a block, query rows of a step
constexpr int FB_TILE = 2 * 128 * 128;    // K, V, Q, dO or dS^T: two 64-column halves of 128 rows x 128 B
constexpr int FB_ROWBLK = 2 * FB_BLK;     // see FaBwdParams::rows
constexpr int FB_SROW = FB_ROWBLK * 4;
constexpr int FB_SMEM = 7 * FB_TILE + 256 + 2 * FB_SROW;
constexpr int FB_ACC_TILE = FB_BLK * FA_D;// floats of one dQ tile
constexpr int FB_DQ_STAGE = FB_TILE / 4;  // per warp: 32 rows x 64 columns of dQ
constexpr int FB_PITCH = 64 + 4;          // floats of a staged accumulator row: eight lanes' 16 bytes fall into different banks
constexpr int FB_STAGED = 32 * FB_PITCH;  // floats that one warp stages: 32 rows, 32 + 32 columns
static_assert(2 * 8 * FB_STAGED * 4 <= 5 * FB_TILE, "staged accumulators lie in the K, V, Q and dO tiles");

struct FaBwdParams {
  // Per query row: log-sum-exp in units of log2 (+inf behind the sequence, which makes every probability of
  // such a row zero) and delta = rowsum(dO * O), [B, Hq, ceil(S / 128)][128 lse | 128 delta]: a block of rows
  // is one aligned copy whatever S is.
  const float* rows;
  // fp32 sums of dQ without the softmax scale, zero on entry, tiles of 128 query rows
  // [B, Hq, ceil(S / 128)][4 x 32 rows][32 groups of 4 columns][32 rows][4]: what a warp whose lanes hold
  // rows reads from TMEM is one contiguous piece of it, staged without bank conflicts.
  float* dq_acc;
  const __nv_bfloat16 *dout, *out;   // [B, S, Hq, 128]
  const float* lse;    // [B, Hq, S]
  __nv_bfloat16* dqkv; // packed [B, S, Hp, 128]
  const float* cos_t;  // [>= S, 64] rotary tables, or null: the gradient is left in rotated coordinates
  const float* sin_t;
  int S, Hkv, rep;
  int split;           // CTAs of a cluster, each with rep / split query heads of the KV group
  float scale, scale_log2;
  BlockOrder order;
};

// Transpose of the rotation by the table row (c, s): (lo, hi) -> (lo c + hi s, hi c - lo s).
__device__ __forceinline__ void rope_bwd_pair(uint32_t& lo, uint32_t& hi, float c, float s) {
  const float a = __uint_as_float(lo), b = __uint_as_float(hi);
  lo = __float_as_uint(a * c + b * s);
  hi = __float_as_uint(b * c - a * s);
}

__device__ __forceinline__ uint4 pack8(const uint32_t* v) {
  return make_uint4(pack_bf16(__uint_as_float(v[0]), __uint_as_float(v[1])), pack_bf16(__uint_as_float(v[2]), __uint_as_float(v[3])),
                    pack_bf16(__uint_as_float(v[4]), __uint_as_float(v[5])), pack_bf16(__uint_as_float(v[6]), __uint_as_float(v[7])));
}

// Eight columns of the rotary tables at one position, if there are tables.
struct RopeCols {
  float4 c[2], s[2];
  __device__ __forceinline__ void load(const FaBwdParams& p, int pos, int col) {
    if (!p.cos_t) return;
    const float4* ct = reinterpret_cast<const float4*>(p.cos_t + static_cast<int64_t>(min(pos, p.S - 1)) * 64 + col);
    const float4* st = reinterpret_cast<const float4*>(p.sin_t + static_cast<int64_t>(min(pos, p.S - 1)) * 64 + col);
    c[0] = __ldg(ct);
    c[1] = __ldg(ct + 1);
    s[0] = __ldg(st);
    s[1] = __ldg(st + 1);
  }
  // dQ and dK: the softmax scale, and the rotation of columns lo and lo + 64 taken back
  __device__ __forceinline__ void apply(const FaBwdParams& p, uint32_t (&lo)[8], uint32_t (&hi)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      lo[i] = __float_as_uint(__uint_as_float(lo[i]) * p.scale);
      hi[i] = __float_as_uint(__uint_as_float(hi[i]) * p.scale);
    }
    if (!p.cos_t) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      rope_bwd_pair(lo[i * 4 + 0], hi[i * 4 + 0], c[i].x, s[i].x);
      rope_bwd_pair(lo[i * 4 + 1], hi[i * 4 + 1], c[i].y, s[i].y);
      rope_bwd_pair(lo[i * 4 + 2], hi[i * 4 + 2], c[i].z, s[i].z);
      rope_bwd_pair(lo[i * 4 + 3], hi[i * 4 + 3], c[i].w, s[i].w);
    }
  }
};

// Stores 8 columns of a gradient row and the same columns + 64.
__device__ __forceinline__ void store_grad8(const FaBwdParams& p, int64_t b, int hp, int pos, int col, const uint32_t (&lo)[8],
                                            const uint32_t (&hi)[8]) {
  uint4* dst = reinterpret_cast<uint4*>(p.dqkv + ((b * p.S + pos) * (p.Hkv * (p.rep + 2)) + hp) * FA_D + col);
  dst[0] = pack8(lo);
  dst[8] = pack8(hi);
}

__device__ __forceinline__ void stage_grad_warp(float* stage, uint32_t acc, int lane) {
  uint32_t lo[32], hi[32];
  tmem_ld_32x32(acc, lo);
  tmem_ld_32x32(acc + 64, hi);
  tmem_ld_wait();
  uint4* mine = reinterpret_cast<uint4*>(stage + lane * FB_PITCH);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    mine[c] = make_uint4(lo[c * 4], lo[c * 4 + 1], lo[c * 4 + 2], lo[c * 4 + 3]);
    mine[8 + c] = make_uint4(hi[c * 4], hi[c * 4 + 1], hi[c * 4 + 2], hi[c * 4 + 3]);
  }
}
// Eight columns of a staged row and the same + 64.
__device__ __forceinline__ void staged8(const float* stage, int row, int col, uint32_t (&lo)[8], uint32_t (&hi)[8]) {
  const uint4* src = reinterpret_cast<const uint4*>(stage + row * FB_PITCH + col);
  const uint4 a = src[0], c = src[1], d = src[8], e = src[9];
  lo[0] = a.x; lo[1] = a.y; lo[2] = a.z; lo[3] = a.w; lo[4] = c.x; lo[5] = c.y; lo[6] = c.z; lo[7] = c.w;
  hi[0] = d.x; hi[1] = d.y; hi[2] = d.z; hi[3] = d.w; hi[4] = e.x; hi[5] = e.y; hi[6] = e.z; hi[7] = e.w;
}

__device__ __forceinline__ float4 fb_ld_cluster(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

template <int R>
__device__ __forceinline__ void regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }

// Four warps with the TMA and the MMA warp, eight compute warps, four warps that reduce dQ. A block is launched with
// 512 x 128 registers, the whole file, and deals them anew: 64 + 2 x 144 + 160 = 4 x 128.
constexpr int FB_THREADS = 512;
// DIRECT: the sequence is one block, so that a CTA has all of a head's dQ: it computes the row statistics itself and stores
// dQ as it is, without the kernels ahead and behind (B2 S128 2 heads 15.4 -> 12.0 us for the three, two launches less).
template <bool DIRECT>
__global__ void __launch_bounds__(FB_THREADS, 1)
    flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ FaBwdParams p, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + FB_TILE;
  uint8_t* sQ = sV + FB_TILE;        // [2 stages]
  uint8_t* sDO = sQ + 2 * FB_TILE;
  uint8_t* sDS = sDO + FB_TILE;
  uint8_t* sDQ = sDS + FB_TILE;      // one FB_DQ_STAGE for each of the four warps
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDQ + FB_TILE);
  uint64_t* k_full = bars;
  uint64_t* v_full = bars + 1;
  uint64_t* q_full = bars + 2;     // [2] Q tile and the step's row statistics
  uint64_t* q_empty = bars + 4;    // [2]
  uint64_t* do_full = bars + 6;
  uint64_t* do_empty = bars + 7;
  uint64_t* s_full = bars + 8;
  uint64_t* p_ready = bars + 9;
  uint64_t* dp_full = bars + 10;
  uint64_t* dv_done = bars + 11;
  uint64_t* ds_ready = bars + 12;
  uint64_t* ds_free = bars + 13;   // dK and dQ of a step have read dS
  uint64_t* dq_full = bars + 14;
  uint64_t* dq_free = bars + 15;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  float* sRow = reinterpret_cast<float*>(sDQ + FB_TILE + 256);   // [2][lse 128 | delta 128]

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x) % p.split;
  int head, jb;   // key block 0 has the most query blocks
  p.order.at(static_cast<int>(blockIdx.x) / p.split, head, jb);
  const int b = head / p.Hkv, g = head - b * p.Hkv;
  const int hp_k = g * (p.rep + 2) + p.rep;
  const int nqb = (p.S + FB_BLK - 1) / FB_BLK;
  const int nq = nqb - jb;              // query blocks at or below the diagonal
  const int heads = p.rep / p.split, r0 = rank * heads;
  const int nsteps = nq * heads;
  if (smem_u32(smem) & 1023) {          // the same in every CTA of a cluster
    if (threadIdx.x == 0) atomicCAS(err, 0, MM_ERR_ATTN_ALIGN);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 16; ++i) mbar_init(&bars[i], i == 9 || i == 12 ? 8 : i == 15 ? 4 : 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQKV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base;          // S^T; P^T (bf16) over columns 0..31 and 64..95 of it
  const uint32_t tDP = tmem_base + 128;   // dP^T, then dQ
  const uint32_t tDV = tmem_base + 256;
  const uint32_t tDK = tmem_base + 384;

  if (warp < 4) {
    regs_fewer<64>();
    if (warp == 0 && elect_one()) {
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int hp, int row) {
        tma_load_4d(dst, map, bar, 0, hp, row, b);
        tma_load_4d(dst + FB_TILE / 2, map, bar, 64, hp, row, b);
      };
      mbar_expect_tx(k_full, FB_TILE);
      load(sK, &tmQKV, k_full, hp_k, jb * FB_BLK);
      bool ok = true;
      for (int n = 0; n < nsteps; ++n) {
        const int st = n & 1;
        const int r = n / nq, i = jb + (n - r * nq);
        const int hq = g * p.rep + r0 + r, hp_q = g * (p.rep + 2) + r0 + r;
        if (!mbar_wait(&q_empty[st], ((n >> 1) & 1) ^ 1, err, MM_ERR_ATTN_WAIT)) { ok = false; break; }
        mbar_expect_tx(&q_full[st], FB_TILE + (DIRECT ? 0 : FB_SROW));
        load(sQ + st * FB_TILE, &tmQKV, &q_full[st], hp_q, i * FB_BLK);
        if constexpr (!DIRECT) {
          const float* src = p.rows + ((static_cast<int64_t>(b) * (p.Hkv * p.rep) + hq) * nqb + i) * FB_ROWBLK;
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           smem_u32(sRow + st * FB_ROWBLK)),
                       "l"(src), "r"(FB_SROW), "r"(smem_u32(&q_full[st]))
                       : "memory");
        }
        if (n == 0) {
          mbar_expect_tx(v_full, FB_TILE);
          load(sV, &tmQKV, v_full, hp_k + 1, jb * FB_BLK);
        }
        if (!mbar_wait(do_empty, (n & 1) ^ 1, err, MM_ERR_ATTN_WAIT)) { ok = false; break; }
        mbar_expect_tx(do_full, FB_TILE);
        load(sDO, &tmDO, do_full, hq, i * FB_BLK);
      }
      if (!ok)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies in flight land before exit
    } else if (warp == 1 && elect_one()) {
      constexpr uint32_t idesc_kk = umma_idesc_bf16(128, 128, false, false);   // K Q^T, V dO^T
      constexpr uint32_t idesc_kn = umma_idesc_bf16(128, 128, false, true);    // P^T dO, dS^T Q
      constexpr uint32_t idesc_nn = umma_idesc_bf16(128, 128, true, true);     // dS K
      // every tile is a K-major operand of the score products and an MN-major one of the others
      auto k_major = [&](const uint8_t* t) { return umma_desc_sw128(smem_u32(t), 16, 1024); };
      auto mn_major = [&](const uint8_t* t) { return umma_desc_sw128(smem_u32(t), FB_TILE / 2, 1024); };
      const uint64_t k_k = k_major(sK), v_k = k_major(sV), q_k = k_major(sQ), do_k = k_major(sDO), ds_k = k_major(sDS);
      const uint64_t k_mn = mn_major(sK), q_mn = mn_major(sQ), do_mn = mn_major(sDO), ds_mn = mn_major(sDS);
      auto scores = [&](uint32_t d, uint64_t a, uint64_t t) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t at = (kk >> 2) * (FB_TILE / 2) + (kk & 3) * 32;
          umma_bf16(d, umma_desc_at(a, at), umma_desc_at(t, at), idesc_kk, kk ? 1u : 0u);
        }
      };
      bool ok = mbar_wait(k_full, 0, err, MM_ERR_ATTN_WAIT) && mbar_wait(&q_full[0], 0, err, MM_ERR_ATTN_WAIT);
      if (ok) {
        tc_fence_after();
        scores(tS, k_k, q_k);
        umma_commit(s_full);
        ok = mbar_wait(v_full, 0, err, MM_ERR_ATTN_WAIT);
      }
      for (int n = 0; n < nsteps && ok; ++n) {
        const int st = n & 1;
        // dP^T, where dQ of the step before has left its columns
        if (!mbar_wait(do_full, n & 1, err, MM_ERR_ATTN_WAIT) || (n > 0 && !mbar_wait(dq_free, (n - 1) & 1, err, MM_ERR_ATTN_WAIT))) break;
        tc_fence_after();
        scores(tDP, v_k, do_k);
        umma_commit(dp_full);
        if (!mbar_wait(p_ready, n & 1, err, MM_ERR_ATTN_WAIT)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)     // dV += P^T dO
          umma_bf16_ts(tDV, tS + (kk >> 2) * 64 + (kk & 3) * 8, umma_desc_at(do_mn, kk * 2048), idesc_kn, (n | kk) ? 1u : 0u);
        umma_commit(dv_done);
        umma_commit(do_empty);
        if (n + 1 < nsteps) {
          // P^T is read: the next scores go over it, ahead of this step's dS
          const int m = n + 1;
          if (!mbar_wait(&q_full[m & 1], (m >> 1) & 1, err, MM_ERR_ATTN_WAIT) || !mbar_wait(dv_done, n & 1, err, MM_ERR_ATTN_WAIT)) break;
          tc_fence_after();
          scores(tS, k_k, umma_desc_at(q_k, (m & 1) * FB_TILE));
          umma_commit(s_full);
        }
        if (!mbar_wait(ds_ready, n & 1, err, MM_ERR_ATTN_WAIT)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)     // dQ = dS K over the columns of dP^T, which has been read
          umma_bf16(tDP, umma_desc_at(ds_mn, kk * 2048), umma_desc_at(k_mn, kk * 2048), idesc_nn, kk ? 1u : 0u);
        umma_commit(dq_full);
        const uint64_t qb = umma_desc_at(q_mn, st * FB_TILE);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)     // dK += dS^T Q
          umma_bf16(tDK, umma_desc_at(ds_k, (kk >> 2) * (FB_TILE / 2) + (kk & 3) * 32), umma_desc_at(qb, kk * 2048), idesc_kn,
                    (n | kk) ? 1u : 0u);
        umma_commit(&q_empty[st]);
        umma_commit(ds_free);
      }
    }
  } else if (warp >= 12) {
    // dQ leaves TMEM as soon as it is complete (the next step's dP^T waits for its columns) and is added to memory by
    // bulk reductions, half a tile at a time through shared memory. As instructions (red.global.add.v4, straight from the
    // registers) the additions held up the load/store unit: B1 S8192 32 / 8 heads 1.72 ms against 1.32.
    regs_more<160>();
    const int q = warp & 3;
    uint8_t* stage = sDQ + q * FB_DQ_STAGE;
    bool ok = true;
    RopeCols rope[4];        // DIRECT: of this lane's columns in the next half of a tile
    if constexpr (DIRECT) {
#pragma unroll
      for (int k = 0; k < 4; ++k) rope[k].load(p, q * 32 + k * 8 + (lane >> 2), (lane & 3) * 8);
    }
    for (int n = 0; n < nsteps; ++n) {
      const int r = n / nq, i = jb + (n - r * nq);
      if (!__all_sync(0xffffffffu, mbar_wait(dq_full, n & 1, err, MM_ERR_ATTN_WAIT))) ok = false;   // uniform: elections follow
      tc_fence_after();
      if constexpr (DIRECT) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t lo[32], hi[32];
          tmem_ld_32x32(tDP + (static_cast<uint32_t>(q * 32) << 16) + h * 32, lo);
          tmem_ld_32x32(tDP + (static_cast<uint32_t>(q * 32) << 16) + 64 + h * 32, hi);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(dq_free);
          }
          __syncwarp();                          // the previous half has been read
          uint4* mine = reinterpret_cast<uint4*>(stage) + lane * 16;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            mine[c ^ (lane & 7)] = make_uint4(lo[c * 4], lo[c * 4 + 1], lo[c * 4 + 2], lo[c * 4 + 3]);
            mine[8 + (c ^ (lane & 7))] = make_uint4(hi[c * 4], hi[c * 4 + 1], hi[c * 4 + 2], hi[c * 4 + 3]);
          }
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int row = k * 8 + (lane >> 2), c0 = (lane & 3) * 2, pos = q * 32 + row;
            const uint4* src = reinterpret_cast<const uint4*>(stage) + row * 16;
            const uint4 a = src[c0 ^ (row & 7)], d = src[(c0 + 1) ^ (row & 7)], e = src[8 + (c0 ^ (row & 7))], f = src[8 + ((c0 + 1) ^ (row & 7))];
            uint32_t l8[8] = {a.x, a.y, a.z, a.w, d.x, d.y, d.z, d.w}, h8[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
            rope[k].apply(p, l8, h8);
            if (ok && pos < p.S) store_grad8(p, b, g * (p.rep + 2) + r0 + r, pos, h * 32 + c0 * 4, l8, h8);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) rope[k].load(p, q * 32 + k * 8 + (lane >> 2), (1 - h) * 32 + (lane & 3) * 8);
        }
        continue;
      }
      float* dst = p.dq_acc + ((static_cast<int64_t>(b) * (p.Hkv * p.rep) + g * p.rep + r0 + r) * nqb + i) * FB_ACC_TILE + q * (FB_ACC_TILE / 4);
      uint32_t v[4][32];
#pragma unroll
      for (int h = 0; h < 4; ++h) tmem_ld_32x32(tDP + (static_cast<uint32_t>(q * 32) << 16) + h * 32, v[h]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_free);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (elect_one()) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the stage has been read
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const uint32_t* w = v[h * 2 + (c >> 3)] + (c & 7) * 4;
          *reinterpret_cast<uint4*>(stage + c * 512 + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (ok && elect_one()) {
          asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst + h * (FB_DQ_STAGE / 4)),
                       "r"(smem_u32(stage)), "r"(FB_DQ_STAGE)
                       : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        __syncwarp();
      }
    }
    if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  } else {
    regs_more<144>();
    // Eight compute warps: two per TMEM lane quarter, each with 64 of the step's 128 query columns.
    const int q = warp & 3, half = (warp - 4) >> 2, t = q * 32 + lane;   // t: key row
    const uint32_t lanes = static_cast<uint32_t>(q * 32) << 16, own = lanes + half * 64;
    bool ok = true;
    for (int n = 0; n < nsteps; ++n) {
      const int st = n & 1;
      const float4* lse = reinterpret_cast<const float4*>(sRow + st * FB_ROWBLK + half * 64);
      const float4* delta = lse + FB_BLK / 4;
      if constexpr (DIRECT) {
        // the step's row statistics: sixteen lanes to a row, under the loads and the first product
        const int row0 = (warp - 4) * 16, hq = g * p.rep + r0 + n, l16 = lane & 15;
        uint4 a[8], c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int row = row0 + k * 2 + (lane >> 4);
          const int64_t at = ((static_cast<int64_t>(b) * p.S + row) * (p.Hkv * p.rep) + hq) * FA_D + l16 * 8;
          a[k] = c[k] = make_uint4(0, 0, 0, 0);
          if (row < p.S) {
            a[k] = *reinterpret_cast<const uint4*>(p.dout + at);
            c[k] = *reinterpret_cast<const uint4*>(p.out + at);
          }
        }
        float* rows = sRow + st * FB_ROWBLK;
        if (lane < 16)
          rows[row0 + lane] = row0 + lane < p.S
                                  ? p.lse[(static_cast<int64_t>(b) * (p.Hkv * p.rep) + hq) * p.S + row0 + lane] * 1.4426950408889634f
                                  : INFINITY;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t aw[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, cw[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
          float sum = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 x = unpack_bf16(aw[j]), y = unpack_bf16(cw[j]);
            sum += x.x * y.x + x.y * y.y;
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          if (l16 == 0) rows[FB_BLK + row0 + k * 2 + (lane >> 4)] = sum;
        }
        // the eight compute warps; a stage's rows are written again two steps on, behind the next step's barrier
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      // ---- P^T
      if (ok && !mbar_wait(&q_full[st], (n >> 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;   // the rows
      if (ok && !mbar_wait(s_full, n & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
      tc_fence_after();
      uint32_t s[2][32];
      tmem_ld_32x32(tS + own, s[0]);
      tmem_ld_32x32(tS + own + 32, s[1]);
      tmem_ld_wait();
#pragma unroll
      for (int c4 = 0; c4 < 16; ++c4) {
        const float4 ls = lse[c4];
        uint32_t* x = s[c4 >> 3] + (c4 & 7) * 4;
        x[0] = __float_as_uint(fast_exp2(__uint_as_float(x[0]) * p.scale_log2 - ls.x));
        x[1] = __float_as_uint(fast_exp2(__uint_as_float(x[1]) * p.scale_log2 - ls.y));
        x[2] = __float_as_uint(fast_exp2(__uint_as_float(x[2]) * p.scale_log2 - ls.z));
        x[3] = __float_as_uint(fast_exp2(__uint_as_float(x[3]) * p.scale_log2 - ls.w));
      }
      if (n % nq == 0) {   // the diagonal block: query row >= key row
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (t > half * 64 + c) s[c >> 5][c & 31] = 0;
      }
      {
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 32; ++c)
          pk[c] = pack_bf16(__uint_as_float(s[c >> 4][(c & 15) * 2]), __uint_as_float(s[c >> 4][(c & 15) * 2 + 1]));
        tmem_st_32x32(tS + own, pk);   // over this warp's own scores
        tmem_st_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      // ---- dS^T (dK and dQ are scaled where they are stored)
      if (ok && !mbar_wait(dp_full, n & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
      tc_fence_after();
      uint8_t* drow = sDS + half * (FB_TILE / 2) + t * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t d[32];
        tmem_ld_32x32(tDP + own + h * 32, d);
        tmem_ld_wait();
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4) {
          const float4 dl = delta[h * 8 + c4];
          const uint32_t* x = s[h] + c4 * 4;
          uint32_t* y = d + c4 * 4;
          y[0] = __float_as_uint(__uint_as_float(x[0]) * (__uint_as_float(y[0]) - dl.x));
          y[1] = __float_as_uint(__uint_as_float(x[1]) * (__uint_as_float(y[1]) - dl.y));
          y[2] = __float_as_uint(__uint_as_float(x[2]) * (__uint_as_float(y[2]) - dl.z));
          y[3] = __float_as_uint(__uint_as_float(x[3]) * (__uint_as_float(y[3]) - dl.w));
        }
        if (h == 0 && n > 0 && ok && !mbar_wait(ds_free, (n - 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(drow + ((h * 4 + ch) ^ (t & 7)) * 16) = pack8(d + ch * 8);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
    }
    // A warp stores 32 rows of dK and dV, columns [32 half, 32 half + 32) and the same of the upper 64 (a rotary pair is
    // 64 columns apart). Lanes hold rows of the accumulators; through shared memory four lanes come to hold 32
    // consecutive columns of a row, which is how gradients and rotary tables are contiguous. The tables are on their
    // way while dV is stored: loaded where they are used they took 4,500 cycles of a block, read by rows 7,000.
    const int row0 = jb * FB_BLK + q * 32;
    // every product is complete: the dK / dV accumulators
    if (ok && !mbar_wait(ds_free, (nsteps - 1) & 1, err, MM_ERR_ATTN_WAIT)) ok = false;
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    float* stage = reinterpret_cast<float*>(smem) + (warp - 4) * 2 * FB_STAGED;
    stage_grad_warp(stage, tDK + lanes + half * 32, lane);
    stage_grad_warp(stage + FB_STAGED, tDV + lanes + half * 32, lane);
    __syncwarp();
    if (p.split == 1) {
      RopeCols rope[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) rope[k].load(p, row0 + k * 8 + (lane >> 2), half * 32 + (lane & 3) * 8);
#pragma unroll
      for (int which = 1; which >= 0; --which)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int row = k * 8 + (lane >> 2), col = (lane & 3) * 8;
          uint32_t lo[8], hi[8];
          staged8(stage + which * FB_STAGED, row, col, lo, hi);
          if (which == 0) rope[k].apply(p, lo, hi);
          if (ok && row0 + row < p.S) store_grad8(p, b, hp_k + which, row0 + row, half * 32 + col, lo, hi);
        }
    }
  }

  if (p.split > 1) {
    cluster_sync();
    if (warp >= 4 && warp < 12) {
      const int rows = FB_BLK / p.split;
      for (int u = static_cast<int>(threadIdx.x) - 128; u < 2 * rows * 8; u += 256) {
        const int which = u / (rows * 8), row = rank * rows + (u >> 3) % rows, col = (u & 7) * 8, pos = jb * FB_BLK + row;
        if (pos >= p.S) continue;
        RopeCols rope;
        if (which == 0) rope.load(p, pos, col);
        const int w = (row >> 5) + (col >> 5) * 4;    // the warp that staged them
        const uint32_t at = smem_u32(reinterpret_cast<float*>(smem) + (w * 2 + which) * FB_STAGED + (row & 31) * FB_PITCH + (col & 31));
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int s = 0; s < p.split; ++s) {
            const float4 v = fb_ld_cluster(at + (c >> 1) * 128 + (c & 1) * 16, s);
            a = make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
          }
          uint32_t* o = (c < 2 ? lo : hi) + (c & 1) * 4;
          o[0] = __float_as_uint(a.x);
          o[1] = __float_as_uint(a.y);
          o[2] = __float_as_uint(a.z);
          o[3] = __float_as_uint(a.w);
        }
        if (which == 0) rope.apply(p, lo, hi);
        store_grad8(p, b, hp_k + which, pos, col, lo, hi);
      }
    }
    cluster_sync();   // nobody leaves while a partner may still read its sums
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Row statistics of the backward pass (FaBwdParams::rows) and the zero-filled dQ accumulator in one pass over
// dO and O: half a warp per (b, s, h) row with 16-byte loads, two rows per half warp in flight. Rows
// [S, 128 ceil(S / 128)) of every head get lse = +inf and delta = 0. Bound by memory: 1 KB in
// (dO, O) and 512 bytes of zeros out per row.
__global__ void flash_bwd_prep_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                      const float* __restrict__ lse, float* __restrict__ rows,
                                      float* __restrict__ dq_acc, int B, int S, int Hq) {
  const int64_t warp_id = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int half = lane >> 4, l16 = lane & 15;
  const int nqb = (S + FB_BLK - 1) / FB_BLK, Sp = nqb * FB_BLK;
  const int64_t total = static_cast<int64_t>(B) * Sp * Hq;
  const int64_t r[2] = {warp_id * 4 + half, warp_id * 4 + 2 + half};   // rows are (b, padded s, h)
  uint4 a[2], c[2];
  int h[2], sidx[2];
  int64_t bidx[2];
  bool live[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int64_t bs = r[k] / Hq;
    h[k] = static_cast<int>(r[k] - bs * Hq);
    bidx[k] = bs / Sp;
    sidx[k] = static_cast<int>(bs - bidx[k] * Sp);
    live[k] = r[k] < total && sidx[k] < S;
    if (r[k] < total) {   // the accumulator has as many rows, in an order of its own
      float4* z = reinterpret_cast<float4*>(dq_acc + r[k] * FA_D);
      z[l16] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[l16 + 16] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (live[k]) {
      const int64_t row = (bidx[k] * S + sidx[k]) * Hq + h[k];
      a[k] = *reinterpret_cast<const uint4*>(dout + row * FA_D + l16 * 8);
      c[k] = *reinterpret_cast<const uint4*>(out + row * FA_D + l16 * 8);
    } else {
      a[k] = c[k] = make_uint4(0, 0, 0, 0);
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t aw[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, cw[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(aw[j]), y = unpack_bf16(cw[j]);
      s += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (l16 == 0 && r[k] < total) {
      float* dst = rows + ((bidx[k] * Hq + h[k]) * nqb + sidx[k] / FB_BLK) * FB_ROWBLK + sidx[k] % FB_BLK;
      dst[0] = live[k] ? lse[(bidx[k] * Hq + h[k]) * S + sidx[k]] * 1.4426950408889634f : INFINITY;
      dst[FB_BLK] = s;
    }
  }
}

// scale * dq_acc -> bf16 query slots of the packed gradient buffer, rotated back when tables are given. A block takes 32
// rows (16 KB, contiguous), turns them around in shared memory and stores them eight lanes to a row, which is how
// gradients and tables are contiguous.
__global__ void __launch_bounds__(256)
    flash_dq_store_kernel(FaBwdParams p) {
  __shared__ float4 tile[32 * 33];      // [row][column group], a row padded by one group
  const int nqb = p.order.nblk, Hq = p.Hkv * p.rep;
  const int tile_id = static_cast<int>(blockIdx.x >> 2), quarter = static_cast<int>(blockIdx.x & 3);
  const int bh = tile_id / nqb, pos0 = (tile_id - bh * nqb) * FB_BLK + quarter * 32;
  const float4* src = reinterpret_cast<const float4*>(p.dq_acc) + (static_cast<int64_t>(tile_id) * 4 + quarter) * (FB_ACC_TILE / 16);
  if (pos0 >= p.S) return;
  RopeCols rope;
  rope.load(p, pos0 + static_cast<int>(threadIdx.x >> 3), static_cast<int>(threadIdx.x & 7) * 8);
  float4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = src[i * 256 + threadIdx.x];
#pragma unroll
  for (int i = 0; i < 4; ++i) tile[(threadIdx.x & 31) * 33 + i * 8 + (threadIdx.x >> 5)] = v[i];
  __syncthreads();
  const int row = threadIdx.x >> 3, part = threadIdx.x & 7, b = bh / Hq, hq = bh - b * Hq, g = hq / p.rep;
  if (pos0 + row >= p.S) return;
  const uint4* t = reinterpret_cast<const uint4*>(tile + row * 33 + part * 2);
  const uint4 a = t[0], c = t[1], d = t[16], e = t[17];
  uint32_t lo[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w}, hi[8] = {d.x, d.y, d.z, d.w, e.x, e.y, e.z, e.w};
  rope.apply(p, lo, hi);
  store_grad8(p, b, g * (p.rep + 2) + hq - g * p.rep, pos0 + row, part * 8, lo, hi);
}

static int packed_map(CUtensorMap* out, const void* base, int B, int S, int H, int box_rows) {
  const uint64_t dims[4] = {static_cast<uint64_t>(FA_D), static_cast<uint64_t>(H), static_cast<uint64_t>(S),
                            static_cast<uint64_t>(B)};
  const uint64_t strides[4] = {0, static_cast<uint64_t>(FA_D) * 2, static_cast<uint64_t>(H) * FA_D * 2,
                               static_cast<uint64_t>(S) * H * FA_D * 2};
  const uint32_t box[4] = {64, 1, static_cast<uint32_t>(box_rows), 1};
  return encode_tmap_bf16(out, base, 4, dims, strides, box, 1);
}

}  // namespace mm

// CTAs of a cluster that share the query heads of one key block. More of them shorten the longest block (all heads
// against the first keys) but each repeats the block's fixed part and the cluster adds its gradients at the end. In steps
// of 128 x 128 (3.4 us in the mean of the fitted shapes; 2.7 us on B1 S8192 32/8 heads): 2 for a block's start and end,
// 1.5 more for a cluster and 0.3 for each of its CTAs (fitted to 150 measured shapes x splits, S 64 to 8192, 1 to 128 KV
// heads, rep 2 to 8; the choice is 0.5 % from the best of them on average, 20 % at most). Where a sequence is one block its
// steps take 4.0 us, with their row statistics, and a cluster costs 1.4 of them whatever its size: B8 S64 32/8 heads 23.1
// us unsplit, 21.5 over two CTAs (21.2 in steps of 64 rows, before), B8 S128 32/8 26.5 | 24.1, B16 S64 32/4 39.2 | 29.8. The blocks of one round last as long as the longest, more than a round as long as the
// chip's share of all of them and one of the shortest, which ends last. Splitting whenever the longest block exceeded
// the chip's share of the steps alone was 15 % from the best: B16 S128 32/8 heads 50 us against 31 unsplit, B2 S1000
// 32/8 heads 108 against 72 over two CTAs.
static int bwd_split(int64_t kv_heads, int rep, int nqb, int sms) {
  int best = 1;
  double best_time = 0;
  for (int s = 1; s <= 8 && rep % s == 0; s *= 2) {
    const double fixed = s == 1 ? 2.0 : nqb == 1 ? 3.4 : 3.5 + 0.3 * s;
    const double blocks = static_cast<double>(kv_heads) * nqb * s, steps = static_cast<double>(kv_heads) * rep * nqb * (nqb + 1) / 2;
    double time = static_cast<double>(nqb) * rep / s + fixed;
    if (blocks > sms) time = std::max(time, (steps + fixed * blocks) / sms + static_cast<double>(rep) / s + fixed);
    if (s == 1 || time < 0.98 * best_time) {
      best = s;
      best_time = time;
    }
  }
  return best;
}

extern "C" {

// 1 when (S, D) can run on the tcgen05 attention kernels.
// Any sequence length: the last tile of a ragged sequence is zero-filled by TMA, masked by
// causality (a row inside the sequence never looks behind it) and not stored.
int mm_flash_attn_supported(int S, int D) { return (D == mm::FA_D && S >= 1) ? 1 : 0; }

// qkv: packed bf16 [B, S, Hkv*(rep+2), 128] (contiguous); out: bf16 [B, S, Hkv*rep, 128];
// lse: fp32 [B, Hkv*rep, S]. Causal, scale 1/sqrt(128).
int mm_flash_attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int Hkv, int rep, int D,
                      cudaStream_t stream) {
  using namespace mm;
  if (!mm_flash_attn_supported(S, D)) return -2;
  DeviceState* ds = device_state();
  if (!ds) return -1;
  const int Hp = Hkv * (rep + 2);
  CUtensorMap tmQ, tmKV;
  int rc = packed_map(&tmQ, qkv, B, S, Hp, FA_BM);
  if (rc) return rc;
  rc = packed_map(&tmKV, qkv, B, S, Hp, FA_BN);
  if (rc) return rc;
  static bool configured[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev]) {
    MM_CUDA_TRY(cudaFuncSetAttribute(flash_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_FWD_SMEM));
    configured[dev] = true;
  }
  FaFwdParams p;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.S = S;
  p.Hkv = Hkv;
  p.rep = rep;
  p.scale_log2 = 1.4426950408889634f / sqrtf(static_cast<float>(D));
  const int nblk = (S + FA_BM - 1) / FA_BM;
  // what a head reads again and again: keys and values, shared by the query heads of a KV group
  p.order = block_order(static_cast<int64_t>(B) * Hkv * rep, static_cast<int64_t>(S) * FA_D * 4 / rep + 1, nblk, 2 * ds->sm_count);
  const unsigned grid = static_cast<unsigned>(p.order.heads) * nblk;
  flash_fwd_kernel<<<grid, FA_THREADS, FA_FWD_SMEM, stream>>>(tmQ, tmKV, p, ds->status);
  MM_LAUNCHED(1);
  return 0;
}

// Floats of the row-statistics scratch of the backward pass (sequences of one block need none).
int64_t mm_flash_attn_bwd_rows(int B, int S, int Hq) {
  const int nqb = (S + mm::FB_BLK - 1) / mm::FB_BLK;
  return nqb <= 1 ? 4 : static_cast<int64_t>(B) * Hq * nqb * mm::FB_ROWBLK;
}

// Floats of the dQ scratch of the backward pass.
int64_t mm_flash_attn_bwd_acc(int B, int S, int Hq) {
  const int nqb = (S + mm::FB_BLK - 1) / mm::FB_BLK;
  return nqb <= 1 ? 4 : static_cast<int64_t>(B) * Hq * nqb * mm::FB_ACC_TILE;
}

// dqkv: packed bf16 gradient buffer, same layout as qkv (every element is written).
// dq_acc, rows: fp32 scratch of mm_flash_attn_bwd_acc and mm_flash_attn_bwd_rows floats.
// cos_t / sin_t: fp32 [>= S, 64] rotary tables of the forward pass, or null. With tables the query
// and key gradients are rotated back as they are stored (position = row of the sequence), which
// replaces a read-modify-write pass over both.
int mm_flash_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv,
                      float* dq_acc, float* rows, const float* cos_t, const float* sin_t, int B, int S, int Hkv, int rep,
                      int D, cudaStream_t stream) {
  using namespace mm;
  if (!mm_flash_attn_supported(S, D)) return -2;
  DeviceState* ds = device_state();
  if (!ds) return -1;
  const int Hp = Hkv * (rep + 2), Hq = Hkv * rep;
  CUtensorMap tmQKV, tmDO;
  int rc = packed_map(&tmQKV, qkv, B, S, Hp, FB_BLK);
  if (rc) return rc;
  rc = packed_map(&tmDO, dout, B, S, Hq, FB_BLK);
  if (rc) return rc;
  static bool configured[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev]) {
    MM_CUDA_TRY(cudaFuncSetAttribute(flash_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM));
    MM_CUDA_TRY(cudaFuncSetAttribute(flash_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM));
    configured[dev] = true;
  }
  const int nqb = (S + FB_BLK - 1) / FB_BLK;
  const int64_t tiles = static_cast<int64_t>(B) * Hq * nqb;
  const bool direct = nqb == 1;
  if (!direct) {
    const int threads = 256;      // four rows per warp
    flash_bwd_prep_kernel<<<static_cast<unsigned>(tiles * (FB_BLK / 32)), threads, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(out), lse, rows, dq_acc, B, S, Hq);
  }
  FaBwdParams p;
  p.rows = rows;
  p.dout = static_cast<const __nv_bfloat16*>(dout);
  p.out = static_cast<const __nv_bfloat16*>(out);
  p.lse = lse;
  p.cos_t = cos_t;
  p.sin_t = sin_t;
  p.dq_acc = dq_acc;
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.S = S;
  p.Hkv = Hkv;
  p.rep = rep;
  p.scale = 1.f / sqrtf(static_cast<float>(D));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.split = bwd_split(static_cast<int64_t>(B) * Hkv, rep, nqb, ds->sm_count);
  // queries and output gradients (bf16) and the dQ sums (fp32) of the KV group's heads
  p.order = block_order(static_cast<int64_t>(B) * Hkv, static_cast<int64_t>(S) * FA_D * 8 * rep, nqb, ds->sm_count / p.split);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.order.heads) * nqb * p.split, 1, 1);
  cfg.blockDim = dim3(FB_THREADS, 1, 1);
  cfg.dynamicSmemBytes = FB_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(p.split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.split > 1 ? 1 : 0;
  MM_CUDA_TRY(cudaLaunchKernelEx(&cfg, direct ? flash_bwd_kernel<true> : flash_bwd_kernel<false>, tmQKV, tmDO, p, ds->status));
  if (!direct) flash_dq_store_kernel<<<static_cast<unsigned>(tiles * 4), 256, 0, stream>>>(p);
  MM_LAUNCHED(direct ? 1 : 3);
  return 0;
}

}  // extern "C"
