// Device helpers of the tcgen05 GEMM kernels: mbarriers, TMA and cp.async copies, tcgen05 instructions and their
// descriptors, and where an epilogue stores.
#pragma once
#include <cuda.h>

#include "hg_gemm_tc.cuh"

namespace hg {

// Where the epilogue stores: `ptr` is [tokens, outputs] of 16-bit elements, or of fp32 when `f32` is set.
// For a row-parallel partial (hg_run_partial) `ptr` is this rank's exchange buffer, `epoch` the device word
// that counts finished exchanges and `parity_bytes` the distance between the two halves of the buffer; the
// half written is the one of exchange `*epoch + 1`.
struct OutTargets {
  void* ptr;
  int f32;
  const int* epoch;
  int64_t parity_bytes;
};

// Builds with -DHG_TRACE record, per CTA, the global timer at sixteen points of the kernel (hg_trace reads them
// back; `bench.py --timeline` prints their distribution over the grid).  Slots: 0 entry, 1 set-up done, 2 dependency
// wait released (TMA thread), 3 first full stage seen by issuer 0, 4-7 issuer 0's commit of its first four units,
// 8/9, 10/11, 12/13 start and end of the first three epilogues (thread 64).  Ordinary builds compile none of it.
#ifdef HG_TRACE
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define HG_STAMP(slot) do { if (p.trace) p.trace[blockIdx.x * 16 + (slot)] = global_timer_ns(); } while (0)
#else
#define HG_STAMP(slot) do { } while (0)
#endif

constexpr int kLoaderThreads = 128;  // weight loaders
constexpr int kQuantThreads = 128;   // activation quantisers (fused quantisation)

// Codes a bounded wait leaves in the status word (times a million, plus the CTA).
enum : int { kErrProducer = 1, kErrMmaFull = 2, kErrMmaAcc = 3, kErrEpilogue = 4, kErrDrain = 5, kErrLoader = 6 };

constexpr long long kWaitLimitCycles = 4000000000ll;  // about 2 s at the boost clock, per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  Returns false when the limit expired or another role of this
// CTA already gave up (abort flag in shared memory).  The clock is only read on
// the slow path, every 256 failed polls (each poll itself blocks in hardware for
// a short, implementation-defined time).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int burst = 0; burst < 256; ++burst)
    if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
#pragma unroll 1
  for (uint32_t spin = 1;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 255u) == 0) {
      if (*abort_flag) return false;
      if (clock64() - start > kWaitLimitCycles) return false;
    }
  }
}

// Wait on a barrier that another CTA of the cluster arrives on: what it wrote before is then visible here.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const long long start = clock64();
#pragma unroll 1
  for (uint32_t spin = 1;; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((spin & 255u) == 0 && (*abort_flag || clock64() - start > kWaitLimitCycles)) return false;
  }
}
// The same waits by a whole warp, with one verdict for all lanes.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)) != 0;
}
__device__ __forceinline__ bool warp_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, abort_flag)) != 0;
}
// True in one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}"
      : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_cp_scales(uint32_t tmem_addr, uint64_t smem_desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_addr), "l"(smem_desc) : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate, uint32_t tmem_sfa, uint32_t tmem_sfb) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n"
      "}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}
__device__ __forceinline__ void tc_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}
// A register filled by a tcgen05.ld issued before the last tc_wait_ld(): passing it through this (empty)
// volatile statement keeps every use behind that wait, however far ahead the load was issued.
__device__ __forceinline__ uint32_t tc_loaded(uint32_t v) {
  asm volatile("" : "+r"(v));
  return v;
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor (tcgen05 format, version 1).
//   bits [0,14) start address >> 4, [16,30) leading byte offset >> 4,
//   [32,46) stride byte offset >> 4, [46,48) version = 1, [61,64) swizzle mode.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  return uint64_t((addr & 0x3ffffu) >> 4) | (uint64_t(lbo >> 4) << 16) | (uint64_t(sbo >> 4) << 32) |
         (uint64_t(1) << 46) | (uint64_t(layout) << 61);
}
constexpr uint32_t kSwizzle128B = 2, kSwizzleNone = 0;

// Instruction descriptor of kind::mxf8f6f4.block_scale:
//   [4,6) B scale id, [7,10) A format (0 E4M3, 5 E2M1), [10,13) B format, [15] A major, [16] B major
//   (0 = K-major), [17,23) N>>3, [23] scale format (1 = UE8M0), [24,29) M>>4, [29,31) A scale id.
__device__ __forceinline__ uint32_t instr_desc(bool a_is_fp4, int n_tile) {
  return (a_is_fp4 ? 5u << 7 : 0u) | (0u << 10) | (uint32_t(n_tile >> 3) << 17) | (1u << 23) |
         (uint32_t(kTileRows >> 4) << 24);
}

__device__ __forceinline__ bool epilogue_all(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.b32 p, %1, 0;\n"
      "barrier.cta.red.and.pred q, 1, 128, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}"
      : "=r"(r)
      : "r"(uint32_t(ok))
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("barrier.cta.sync 1, 128;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ void scatter_store(const OutTargets& out, char* base, int64_t index, float v) {
  if (out.f32) reinterpret_cast<float*>(base)[index] = v;
  else reinterpret_cast<uint16_t*>(base)[index] = from_float<T>(v);
}

// Start of the output this launch writes: the plain output, or the half of the exchange buffer that belongs
// to the coming exchange.  Read after pdl_wait(): the word is advanced by the kernel that ends the previous exchange.
__device__ __forceinline__ char* out_base(const OutTargets& out) {
  char* base = static_cast<char*>(out.ptr);
  if (!out.epoch) return base;
  const int e = *reinterpret_cast<const volatile int*>(out.epoch) + 1;
  return base + int64_t(e & 1) * out.parity_bytes;
}

// 8-byte asynchronous copy global -> shared; src_bytes = 0 writes zeros instead.
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// One arrival on `bar` once every cp.async this thread issued so far has landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

}  // namespace hg
