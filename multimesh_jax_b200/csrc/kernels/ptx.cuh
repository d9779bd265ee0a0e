// Thin inline-PTX wrappers for the Blackwell (sm_100a) execution model:
// mbarriers with bounded waits, TMA tensor copies, tcgen05 tensor-core MMA
// with TMEM accumulators, and system-scope flag accesses for peer memory.
//
// Every wait in this header is bounded by wall-clock time (the global timer): when the
// limit runs out it records an error code in a caller-supplied global status word and
// returns false so the kernel can unwind (free TMEM, return) instead of spinning forever.
// The limit lives next to the status word (`status_wait_limit_ns`), so the host sets it per
// device. Once a status word is non-zero every later wait gives up at its first check: the
// step that saw the expiry has failed anyway, and the rest of its kernels must drain in
// milliseconds, not one time limit each. The host reads and clears the word when the step's
// results are awaited and reports the failure there.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mm {

#ifndef MM_SPIN_LIMIT
#define MM_SPIN_LIMIT (1u << 22)   // poll bound of the few waits that have no status word
#endif
#ifndef MM_DEFAULT_WAIT_NS
#define MM_DEFAULT_WAIT_NS 20000000000ull   // used when the status block carries no limit
#endif

// Error codes written to the kernel's status word.
enum : int {
  MM_OK = 0,
  MM_ERR_WAIT_FULL = 1,      // consumer gave up waiting for a TMA stage
  MM_ERR_WAIT_EMPTY = 2,     // producer gave up waiting for a free stage
  MM_ERR_WAIT_TMEM_FULL = 3, // epilogue gave up waiting for the accumulator
  MM_ERR_WAIT_TMEM_EMPTY = 4,// MMA warp gave up waiting for a drained accumulator
  MM_ERR_WAIT_PEER = 5,      // a peer flag never reached the expected value
  MM_ERR_BOUNDS = 6,         // a checked index was out of range
};

// Checked build (-DMM_CHECKED, the stand-in for a memory checker on machines where none may
// run): indices that come from run-time data - row blocks and owners of the fused collectives,
// chunk decoding of the reshard kernel, token ids - are verified before the access that uses
// them. A violation records MM_ERR_BOUNDS in the status word and *skips* the access; nothing
// traps. In the normal build the macros vanish.
#ifdef MM_CHECKED
#define MM_CHECK_OR(cond, err, action)                                     \
  do {                                                                     \
    if (!(cond)) {                                                         \
      if (err) atomicCAS((err), 0, static_cast<int>(mm::MM_ERR_BOUNDS));   \
      action;                                                              \
    }                                                                      \
  } while (0)
#else
#define MM_CHECK_OR(cond, err, action) ((void)0)
#endif

__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// The status block of a device is 64 bytes: word 0 is the status, bytes 8..15 hold the time limit
// of peer waits in nanoseconds (0: the default).
__device__ __forceinline__ unsigned long long status_wait_limit_ns(const int* err) {
  if (!err) return MM_DEFAULT_WAIT_NS;
  const unsigned long long v = *reinterpret_cast<const volatile unsigned long long*>(err + 2);
  return v ? v : MM_DEFAULT_WAIT_NS;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a fully active warp. The branches that issue TMA, tcgen05.mma and tcgen05.commit are
// taken under this predicate and a warp-uniform warp index (below), because only then does the compiler
// know that a single thread executes them: under `lane == 0` it guards every such instruction for a
// divergent warp, and four MMAs with their commit took 380 cycles to issue instead of 80 - more than the
// tensor cores need for them.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(pred));
  return pred != 0;
}

// Index of this thread's warp in its block, known to be the same in every lane.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0); }

// Barrier over all threads of a cluster; what they wrote before it is visible behind it. The aligned instructions
// want every warp whole, and callers come out of loops and branches that lanes leave one by one.
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Orders generic-proxy accesses (plain loads / stores) with async-proxy accesses (TMA) in all
// state spaces: needed when a TMA load reads global memory that plain stores just wrote.
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false (and records `code`) when the limit is reached. The limit is twice
// that of a peer wait: a role that waits for another role which itself waits for a peer must
// not give up first, or the status would name the wrong cause.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
  unsigned long long t0 = 0, limit = 0;
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i > 128) __nanosleep(64);
    if ((i & 1023) == 1023) {
      // once any wait has expired, the others give up at once
      if (err && *reinterpret_cast<volatile int*>(err) != 0) return false;
      if (t0 == 0) {
        t0 = global_timer_ns();
        limit = 2 * status_wait_limit_ns(err);
      } else if (global_timer_ns() - t0 > limit) {
        break;
      }
    }
  }
  if (err) atomicCAS(err, 0, code);
  return false;
}

// --------------------------------------------------------------------- TMA
// 2-D tiled load, global -> shared, completion signalled on an mbarrier.
// `x` is the innermost coordinate: x * element_size must be a multiple of 16.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ----------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; one thread issues for the CTA.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with A in tensor memory: lane = row of A, a 32-bit column holds two neighbouring elements of K.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t of the warp receives lane
// (base_lane + t), columns [col, col + 32).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15,"
      " %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31},"
      " [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Counterpart store: thread t of the warp writes lane (base_lane + t), columns [col, col + 32).
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0],"
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16,"
      " %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
      "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Shared-memory matrix descriptor for a 128-byte-swizzled operand tile.
//  K-major  : rows of 64 bf16 (128 B); 8-row groups 1024 B apart (SBO).
//  MN-major : 64 MN-elements (128 B) contiguous per K row; groups of 8 K rows
//             are `sbo` bytes apart; successive 64-wide MN blocks `lbo` apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes,
                                                    uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);        // start address  [0,14)
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;  // leading offset [16,30)
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;  // stride offset  [32,46)
  d |= static_cast<uint64_t>(1) << 46;                          // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                          // SWIZZLE_128B
  return d;
}
// The descriptor of the same tile `bytes` further on in shared memory (a multiple of 16; the address
// field holds all of an SM's shared memory, so the addition never carries out of it).
__device__ __forceinline__ uint64_t umma_desc_at(uint64_t desc, uint32_t bytes) { return desc + (bytes >> 4); }
// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
  return (1u << 4)                          // D format: F32
         | (1u << 7)                        // A format: BF16
         | (1u << 10)                       // B format: BF16
         | (static_cast<uint32_t>(a_mn) << 15) | (static_cast<uint32_t>(b_mn) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// -------------------------------------------------- peer / system-scope flags
__device__ __forceinline__ void st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int atom_add_release_sys(int* p, int v) {
  int old;
  asm volatile("atom.add.release.sys.global.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
// Wait until *p >= target, for at most the device's peer-wait time limit. Returns false on expiry.
__device__ __forceinline__ bool wait_flag_ge(const int* p, int target, int* err) {
  unsigned long long t0 = 0, limit = 0;
  for (uint32_t i = 0;; ++i) {
    if (ld_acquire_sys(p) >= target) return true;
    if (i > 32) __nanosleep(100);
    if ((i & 255) == 255) {
      if (err && *reinterpret_cast<volatile int*>(err) != 0) return false;
      if (t0 == 0) {
        t0 = global_timer_ns();
        limit = status_wait_limit_ns(err);
      } else if (global_timer_ns() - t0 > limit) {
        break;
      }
    }
  }
  if (err) atomicCAS(err, 0, MM_ERR_WAIT_PEER);
  return false;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

}  // namespace mm
