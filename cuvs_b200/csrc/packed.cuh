// Register-level helpers that several kernels share: two floats in one 64-bit register (one packed instruction for
// both), the three-input minimum and maximum, and a loop whose counter is a compile-time constant.
#pragma once

#include <cstdint>
#include <type_traits>

namespace cuvs_b200 {

__device__ __forceinline__ uint64_t dup2(float x)
{
  uint64_t v;
  asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
  return v;
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi)
{
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
// four floats of shared memory as two pairs (volatile: asynchronous copies write them)
__device__ __forceinline__ void lds128(uint32_t a, uint64_t& x, uint64_t& y)
{
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ float lo2(uint64_t v)
{
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo;
}
__device__ __forceinline__ float hi2(uint64_t v)
{
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return hi;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b)
{
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a * b: the first term of a sum that starts from +0 (fma(a, a, +0) rounds to the same value, and
// a square is never -0), without materialising a zero register pair
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// fn(std::integral_constant<uint32_t, i>) for i = 0 .. kN - 1
template <uint32_t kN, uint32_t kI = 0, typename Fn>
__device__ __forceinline__ void static_for(Fn&& fn)
{
  if constexpr (kI < kN) {
    fn(std::integral_constant<uint32_t, kI>{});
    static_for<kN, kI + 1>(fn);
  }
}

}  // namespace cuvs_b200
