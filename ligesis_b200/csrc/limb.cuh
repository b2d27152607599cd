// Radix-8, -4 and -2 DFTs on 24-bit limbs, and the lazy values between them.
//
// 2 has order 192 mod p (2^96 = -1), so the order-8 root is 2^120 = -2^24.  A value held as four
// signed 32-bit limbs at 2^0, 2^24, 2^48, 2^72 is multiplied by any 8th root of unity by renaming
// and negating limbs, and sums of eight values never leave 28 bits: a radix-8 DFT is plain 32-bit
// adds, with no carries, no corrections and no shifts.  Only its outputs are brought back to 64
// bits (limb_pack), to any representative below 2^64; limb_unpack takes any.  On sm_100, where an
// instruction with a carry issues at half rate, a radix-8 with unpack and pack measured 34.5 issue
// slots per value against 45.7 on canonical 64-bit values with shifts, and 64.8 against 80.5 with
// a twiddle product behind it.
#pragma once
#include "gl64.cuh"

namespace lgs {

struct Limbs {
  int32_t l[4];
};

#ifdef __CUDACC__
// 24 + 24 + 16 bits of any 64-bit value.
__device__ __forceinline__ Limbs limb_unpack(u64 x) {
  const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
  Limbs y;
  y.l[0] = (int32_t)(lo & 0xffffff);
  y.l[1] = (int32_t)(__funnelshift_r(lo, hi, 24) & 0xffffff);
  y.l[2] = (int32_t)(hi >> 16);
  y.l[3] = 0;
  return y;
}
// (a, b) <- (a + 2^(24 R) b, a - 2^(24 R) b).
template <int R>
__device__ __forceinline__ void limb_bfly(Limbs& a, Limbs& b) {
  Limbs s, d;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = (i - R) & 7;  // the limb of b that lands on limb i, negated if t >= 4
    const int32_t x = t >= 4 ? -b.l[t & 3] : b.l[t & 3];
    s.l[i] = a.l[i] + x;
    d.l[i] = a.l[i] - x;
  }
  a = s;
  b = d;
}
// Makes a DFT output's limbs positive: 0 mod p as a whole, each limb above 8 (2^24 - 1), limb 1 by
// more than 2^23 (limb_pack's difference stays positive).
constexpr int32_t LIMB_OFF0 = 0x8000809, LIMB_OFF1 = 0x8f7fef8, LIMB_OFF2 = 0x800fff7,
                  LIMB_OFF3 = 0x8000000;
__device__ __forceinline__ void limb_offset(Limbs& a) {
  a.l[0] += LIMB_OFF0, a.l[1] += LIMB_OFF1, a.l[2] += LIMB_OFF2, a.l[3] += LIMB_OFF3;
}
// 2^(24 R) x.
template <int R>
__device__ __forceinline__ Limbs limb_rot(const Limbs& x) {
  Limbs y;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = (i - R) & 7;
    y.l[i] = t >= 4 ? -x.l[t & 3] : x.l[t & 3];
  }
  return y;
}
// Natural-order radix-R DFTs (radix-2 DIT on bit-reversed inputs) of unpacked values, R = 2, 4, 8:
// w_4 = 2^48; w_8 = 2^120, w_8^2 = 2^48, w_8^3 = 2^168.  ZH (R = 8): the upper half of the inputs
// is zero and not read.  The outputs' limbs are signed, at most 8 (2^24 - 1) in absolute value.
template <int R, bool ZH = false>
__device__ __forceinline__ void limb_dft(Limbs (&v)[R]) {
  static_assert(R == 8 || !ZH, "only the first radix-8 of a padded row has zeros");
  if constexpr (R == 2) {
    limb_bfly<0>(v[0], v[1]);
  } else if constexpr (R == 4) {
    Limbs a0 = v[0], a1 = v[2], a2 = v[1], a3 = v[3];
    limb_bfly<0>(a0, a1);
    limb_bfly<0>(a2, a3);
    limb_bfly<0>(a0, a2);
    limb_bfly<2>(a1, a3);
    v[0] = a0, v[1] = a1, v[2] = a2, v[3] = a3;
  } else {
    Limbs a0 = v[0], a1 = v[4], a2 = v[2], a3 = v[6], a4 = v[1], a5 = v[5], a6 = v[3], a7 = v[7];
    if constexpr (ZH) {
      a1 = a0, a3 = a2, a5 = a4, a7 = a6;
    } else {
      limb_bfly<0>(a0, a1);
      limb_bfly<0>(a2, a3);
      limb_bfly<0>(a4, a5);
      limb_bfly<0>(a6, a7);
    }
    limb_bfly<0>(a0, a2);
    limb_bfly<2>(a1, a3);
    limb_bfly<0>(a4, a6);
    limb_bfly<2>(a5, a7);
    limb_bfly<0>(a0, a4);
    limb_bfly<5>(a1, a5);
    limb_bfly<2>(a2, a6);
    limb_bfly<7>(a3, a7);
    v[0] = a0, v[1] = a1, v[2] = a2, v[3] = a3, v[4] = a4, v[5] = a5, v[6] = a6, v[7] = a7;
  }
}
// A DFT's output V = l0 + l1 2^24 + l2 2^48 + l3 2^72 mod p, some representative below 2^64: with
// the offset the limbs are positive, below 2^28.2, and l1 >= 2^23.  2^72 = 2^40 - 2^8, so with u =
// l2 + (l3 >> 8) and the low byte of l3 put at 2^40, V = l0 + (l1 - (l3 >> 16)) 2^24 -
// (l3 mod 2^16) 2^8 + Y 2^32, Y = u 2^16 + (l3 mod 2^8) 2^8 = y0 + y1 2^32, and Y 2^32 = y0 2^32 +
// y1 (2^32 - 1).  Everything but y0 2^32 sums to a positive number below 2^54, so there is one
// carry out of 64 bits, and its 2^32 - 1 cannot carry again.
__device__ __forceinline__ u64 limb_pack(Limbs x) {
  limb_offset(x);
  const uint32_t l0 = x.l[0], l1 = x.l[1], l2 = x.l[2], l3 = x.l[3];
  const uint32_t u = l2 + (l3 >> 8), y0 = (u << 16) | ((l3 & 0xff) << 8), y1 = u >> 16;
  const uint32_t b = l1 - (l3 >> 16), e = (l3 & 0xffff) << 8;
  u64 a;
  asm("mad.wide.u32 %0, %1, 0x1000000, %2;" : "=l"(a) : "r"(b), "l"((u64)l0));
  uint32_t v0, v1;
  asm("{\n\t.reg .u32 h, c, g;\n\t"
      "add.u32 h, %3, %6;\n\t"
      "add.cc.u32 h, h, %5;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "add.u32 g, %6, %4;\n\t"
      "add.u32 g, g, c;\n\t"
      "sub.cc.u32 %0, %2, g;\n\t"
      "subc.u32 %1, h, 0;\n\t"
      "add.u32 %1, %1, c;\n\t}"
      : "=&r"(v0), "=&r"(v1)
      : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"(e), "r"(y0), "r"(y1));
  return gl_pack(v0, v1);
}
// x 2^R mod p for any 64-bit x and R < 24, some representative below 2^64: the bits t shifted out
// count t (2^32 - 1), which carries once at most.
template <unsigned R>
__device__ __forceinline__ u64 shl_lazy(u64 x) {
  if constexpr (R == 0) {
    return x;
  } else {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    const uint32_t lo = x0 << R, mid = __funnelshift_l(x0, x1, R), t = x1 >> (32 - R);
    uint32_t v0, v1;
    asm("{\n\t.reg .u32 h, g, c;\n\t"
        "add.cc.u32 h, %3, %4;\n\t"
        "addc.u32 g, %4, 0;\n\t"
        "sub.u32 c, g, %4;\n\t"
        "sub.cc.u32 %0, %2, g;\n\t"
        "subc.u32 %1, h, 0;\n\t"
        "add.u32 %1, %1, c;\n\t}"
        : "=&r"(v0), "=&r"(v1)
        : "r"(lo), "r"(mid), "r"(t));
    return gl_pack(v0, v1);
  }
}
// limb_pack(x) 2^S for a compile-time S (any power of two: order 192).
template <unsigned S>
__device__ __forceinline__ u64 limb_pack_shl(const Limbs& x) {
  constexpr unsigned s = S % 192;
  return shl_lazy<s % 24>(limb_pack(limb_rot<s / 24>(x)));
}
// x y mod p for any 64-bit x, y: some representative below 2^64.
__device__ __forceinline__ u64 gl_mul_lazy(u64 x, u64 y) {
#ifdef __CUDA_ARCH__
  uint32_t r[4];
  gl_mul_wide(x, y, r);
  return gl_reduce_lazy(r[0], r[1], r[2], r[3], 0);
#else
  return 0;
#endif
}
// v <- its natural-order R-point DFT; any representatives in, some representatives out.
template <int R>
__device__ __forceinline__ void dft_lazy(u64 (&v)[R]) {
  Limbs x[R];
#pragma unroll
  for (int i = 0; i < R; ++i) x[i] = limb_unpack(v[i]);
  limb_dft<R>(x);
#pragma unroll
  for (int i = 0; i < R; ++i) v[i] = limb_pack(x[i]);
}
#endif  // __CUDACC__

}  // namespace lgs
