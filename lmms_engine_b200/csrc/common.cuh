// Shared device-side building blocks for the sm_100a kernels of this engine:
// mbarrier / TMA / tcgen05 PTX wrappers, bounded waits, bf16 helpers.
//
// Every wait in this file is bounded: a spin that runs out of its cycle budget
// raises a kernel-wide abort word (in shared memory) and a status word in global
// memory, after which every role leaves its loop, the CTA re-converges, frees
// its TMEM and returns.  The host reads the status word and raises.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr long long kWaitCycleLimit = 4000000000LL;  // ~2 s at 1.9 GHz

enum KernelStatus : int {
  kStatusOk = 0,
  kStatusBarrierTimeout = 1,
  kStatusBadShape = 2,
  kStatusPeerTimeout = 3,
  kStatusOverflow = 4,
  kStatusBadIndex = 5,
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t elect_one_sync() {
  uint32_t pred = 0;
  asm volatile(
      "{\n"
      ".reg .b32 rx;\n"
      ".reg .pred px;\n"
      "elect.sync rx|px, %1;\n"
      "selp.u32 %0, 1, 0, px;\n"
      "}\n"
      : "=r"(pred)
      : "r"(0xffffffffu));
  return pred;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  `abort_word` lives in shared memory and is raised by whichever
// role first runs out of budget; everybody else sees it within 64 polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_word,
                                          long long limit = kWaitCycleLimit) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  for (uint32_t i = 1;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 0u) {
      if (*abort_word) return false;
      if (clock64() - t0 > limit) {
        *abort_word = 1;
        return false;
      }
    }
  }
}

// ---------------------------------------------------------------- cross-GPU flags (peer-mapped memory)
// Counters only grow; a waiter compares with wrap-around arithmetic.  Bounded like every wait here.
__device__ __forceinline__ bool flag_wait_ge(const uint32_t* flag, uint32_t target, long long limit,
                                             volatile int* abort_word) {
  const long long t0 = clock64();
  for (uint32_t i = 1;; ++i) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (static_cast<int>(v - target) >= 0) return true;
    if ((i & 15u) == 0u) {
      if (*abort_word) return false;
      if (clock64() - t0 > limit) {
        *abort_word = 1;
        return false;
      }
    }
    __nanosleep(64);
  }
}
__device__ __forceinline__ void flag_add_release(uint32_t* flag, uint32_t v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(flag), "r"(v) : "memory");
}
__device__ __forceinline__ void bar_sync_named(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// ---------------------------------------------------------------- TMA (never multicast)
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]; one thread issues.
__device__ __forceinline__ void umma_bf16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once every previously issued tcgen05.mma of this thread has retired.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major bf16 tile whose rows are 128 bytes
// (64 bf16) wide and stored with the 128-byte swizzle that a TMA box of 64 elements
// produces.  Rows are grouped by eight into 1024-byte swizzle atoms, so the stride
// between 8-row groups (SBO) is 1024 bytes; the leading-dimension offset is unused
// for swizzled K-major operands.  `smem_addr` must be 1024-byte aligned for k = 0;
// stepping along K inside the atom adds the raw byte offset (32 bytes per 16 bf16).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);  // start address, 16-byte units
  d |= static_cast<uint64_t>(1) << 16;                       // LBO (ignored for SW128 K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;               // SBO = 1024 bytes
  d |= static_cast<uint64_t>(1) << 46;                       // descriptor version for sm_100
  d |= static_cast<uint64_t>(2) << 61;                       // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16 with bf16 A/B (both K-major) and fp32 D.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4)                                   // D format fp32
         | (1u << 7)                                 // A format bf16
         | (1u << 10)                                // B format bf16
         | (static_cast<uint32_t>(n >> 3) << 17)     // N / 8
         | (static_cast<uint32_t>(m >> 4) << 24);    // M / 16
}
// Same, but B is MN-major (bit 16) and/or A is MN-major (bit 15).
__host__ __device__ constexpr uint32_t umma_idesc_bf16_major(int m, int n, int a_mn, int b_mn) {
  return umma_idesc_bf16(m, n) | (static_cast<uint32_t>(a_mn) << 15) | (static_cast<uint32_t>(b_mn) << 16);
}

// ---------------------------------------------------------------- packed-document bounds
// A document [start, start + len) of a packed stream must lie inside the tensor it indexes.  Kernels
// that derive row addresses from cu_seqlens call this for the document they were assigned; a table
// that reaches past the tensor raises kStatusBadShape and the CTA does no work instead of writing
// out of bounds.
__device__ __forceinline__ bool doc_in_bounds(int start, int len, int total, int* status) {
  if (start >= 0 && len >= 0 && start + len <= total) return true;
  if (status != nullptr) atomicExch(status, kStatusBadShape);
  return false;
}

// Block `item` of a packed stream whose documents (boundaries cu_a) are cut into blocks of `block` rows, counted over the
// documents in order or, with `from_end`, backwards from the last block of the last document.  One whole warp calls it;
// work[0..5] = document, first row of the block inside it, its length in a and in b, its start in a and in b, or work[0] = -1
// when the stream has fewer blocks.  Thirty-two documents per step: a CTA of a small document lasts a few microseconds, and
// walking 48 to 370 boundaries with one thread cost as much again.
__device__ __forceinline__ void find_block(const int* cu_a, const int* cu_b, int n_docs, int block, int item, bool from_end,
                                           int total_a, int total_b, int* work, int* status) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) work[0] = -1;
  __syncwarp();
  for (int base = 0; base < n_docs; base += 32) {
    const int i = base + lane;
    const int d = from_end ? n_docs - 1 - i : i;
    int lo = 0, len = 0;
    if (i < n_docs) {
      lo = cu_a[d];
      len = cu_a[d + 1] - lo;
    }
    const int nb = len > 0 ? (len + block - 1) / block : 0;
    int sum = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    const bool here = item >= sum - nb && item < sum;
    if (here) {
      const int b = item - (sum - nb);
      work[1] = (from_end ? nb - 1 - b : b) * block;
      work[2] = len;
      work[4] = lo;
      work[5] = cu_b[d];
      work[3] = cu_b[d + 1] - work[5];
      const bool ok = doc_in_bounds(lo, len, total_a, status) && doc_in_bounds(work[5], work[3], total_b, status);
      work[0] = ok ? d : -1;
    }
    if (__any_sync(0xffffffffu, here)) return;
    item -= __shfl_sync(0xffffffffu, sum, 31);
  }
}

// ---------------------------------------------------------------- index bounds
// Rows addressed through an index table (routing tables, gather / scatter maps) are checked against the tensor they
// index: an index past the end raises kStatusBadIndex and the access is skipped.  The check is one compare per row and
// stays on in every build.  B200_DEBUG_BOUNDS (the debug build of the native libraries) switches on the checks that cost
// a compare per ELEMENT or an extra load, through B200_DBG_INDEX.
__device__ __forceinline__ bool index_in_bounds(long idx, long limit, int* status) {
  if (idx < limit) return true;
  if (status != nullptr) atomicExch(status, kStatusBadIndex);
  return false;
}
#ifdef B200_DEBUG_BOUNDS
#define B200_DBG_INDEX(idx, limit, status) index_in_bounds((idx), (limit), (status))
#else
#define B200_DBG_INDEX(idx, limit, status) true
#endif

// ---------------------------------------------------------------- index arithmetic
// i = q * d + r.  A 64-bit division is about a hundred instructions; flat indices nearly always fit 32 bits (`narrow`, the same
// for the whole launch), and the passes that split one per 16 bytes were bound by it rather than by memory.
__device__ __forceinline__ void split_index(long i, int d, bool narrow, long& q, int& r) {
  if (narrow) {
    const unsigned u = static_cast<unsigned>(i), v = u / static_cast<unsigned>(d);
    q = v;
    r = static_cast<int>(u - v * static_cast<unsigned>(d));
  } else {
    q = i / d;
    r = static_cast<int>(i - q * d);
  }
}
__device__ __forceinline__ bool fits32(long n) { return n < (1L << 31); }

// ---------------------------------------------------------------- misc numeric helpers
// 2^x on the special-function unit, one instruction (exp2f() adds a range fix-up for denormal results that a softmax does
// not need): 2^-inf = +0.
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace b200
