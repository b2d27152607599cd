// Sums of many field values through 22-bit limbs, for the sumcheck kernels.
#pragma once
#include "gl64.cuh"

namespace lgs {

// A value's coordinates split into 22 + 22 + 20 bits; limbs of up to 2^10 values add up in 32 bits
// without carries, so a warp's sum is six integer reductions and its CTA's six shared atomics.
__device__ __forceinline__ void limbs22(ef2 v, uint32_t (&l)[6]) {
  constexpr uint32_t M = (1u << 22) - 1;
  l[0] = (uint32_t)v.c0 & M, l[1] = (uint32_t)(v.c0 >> 22) & M, l[2] = (uint32_t)(v.c0 >> 44);
  l[3] = (uint32_t)v.c1 & M, l[4] = (uint32_t)(v.c1 >> 22) & M, l[5] = (uint32_t)(v.c1 >> 44);
}
__device__ __forceinline__ u64 from_limbs22(const uint32_t* l) {
  // l0 + l1 2^22 + l2 2^44 < 2^77: the top limb as u 2^32 with u = l2 2^12
  const u64 a = (u64)l[0] + ((u64)l[1] << 22), u = (u64)l[2] << 12;
  const u64 lo = a + (u << 32);
  return gl_reduce(lo, (u >> 32) + (lo < a ? 1 : 0));
}
// Adds the warp's 32 values to acc[0..6).
__device__ __forceinline__ void warp_add(ef2 v, uint32_t* acc, unsigned lane) {
  uint32_t l[6], mine = 0;
  limbs22(v, l);
#pragma unroll
  for (unsigned i = 0; i < 6; ++i) {
    const uint32_t s = __reduce_add_sync(0xffffffffu, l[i]);
    if (lane == i) mine = s;
  }
  if (lane < 6) atomicAdd(acc + lane, mine);
}
__device__ __forceinline__ ef2 acc_value(const uint32_t* acc) {
  return ef_make(from_limbs22(acc), from_limbs22(acc + 3));
}

}  // namespace lgs
