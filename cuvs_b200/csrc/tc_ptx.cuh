// PTX wrappers shared by the tensor-core kernels: mbarriers with bounded waits, TMA loads, tcgen05.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace cuvs_b200 {

enum { ERR_NONE = 0, ERR_TIMEOUT = 1 };
constexpr uint32_t kSpinLimit = 1u << 21;  // bounded waits (each try_wait sleeps up to ~1 us)

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
  return uint32_t(__cvta_generic_to_shared(p));
}
// One lane of a converged warp.  tcgen05 instructions take their operands from uniform registers: issued under this predicate
// by a warp that goes through its loops as a whole they cost a few clocks, in the branch of a given lane (`lane == 0`) some
// hundred each, for then the compiler cannot know that one thread is there.
__device__ __forceinline__ bool elect_one()
{
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait: false on time-out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit)
{
  for (uint32_t it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
    if (done) { return true; }
  }
  return false;
}
// The same for a whole warp, with one answer for all of it.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, uint32_t limit)
{
  return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, limit));
}
// A batch whose tensor-core pass timed out, counted in the handle's pinned word: by one thread of the kernel behind that
// pass (the kernels of a handle run one after the other).
__device__ __forceinline__ void count_timeout(uint32_t* word)
{
  volatile uint32_t* w = word;
  *w                   = *w + 1u;
  __threadfence_system();
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x,
                                            int y)
{
  asm volatile(
    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
    ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
    : "memory");
}
// `bytes` (a multiple of 16) from 16-byte aligned global memory
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// generic-proxy writes of shared memory become visible to the tensor core and to TMA
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tc_mma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                            uint32_t idesc, uint32_t accumulate)
{
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "setp.ne.b32 p, %4, 0;\n\t"
    "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
    ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
    : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                           uint32_t idesc, uint32_t accumulate)
{
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "setp.ne.b32 p, %4, 0;\n\t"
    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
    ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
    : "memory");
}
// Shared-memory matrix descriptor of a K-major tile stored as rows of 128 bytes (64 halfs) with the
// 128-byte swizzle: 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr)
{
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3FFFFu) >> 4);  // start address, 16-byte units
  d |= uint64_t(1) << 16;                  // leading byte offset (unused for swizzled K-major)
  d |= uint64_t(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= uint64_t(1) << 46;                  // descriptor version of this architecture
  d |= uint64_t(2) << 61;                  // 128-byte swizzle
  return d;
}
// Low word of the descriptor above; its high word is the same for every tile.
__device__ __forceinline__ uint32_t desc_sw128_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
// One step of 16 halfs with descriptors given by their low words: few instructions in front of every MMA, since the one
// thread that issues them shares its scheduler with busy epilogue warps.
template <bool kAccumulate>
__device__ __forceinline__ void tc_mma_f16_lo(uint32_t tmem_d, uint32_t lo_a, uint32_t lo_b, uint32_t idesc)
{
  constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29);
  asm volatile(
    "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
    "setp.ne.b32 p, %5, 0;\n\t"
    "mov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\t"
    "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
    ::"r"(tmem_d), "r"(lo_a), "r"(lo_b), "r"(idesc), "r"(kHi), "n"(kAccumulate ? 1 : 0)
    : "memory");
}
// The load alone; tmem_ld_wait makes its registers valid.
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32])
{
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
      "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
      "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
      "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
    : "r"(taddr)
    : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32])
{
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  // the registers pass through these statements so that nothing that uses them moves above the wait
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]),
                      "+r"(r[i + 6]), "+r"(r[i + 7]));
  }
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
  tmem_ld32_async(taddr, r);
  tmem_ld_wait(r);
}

}  // namespace cuvs_b200
