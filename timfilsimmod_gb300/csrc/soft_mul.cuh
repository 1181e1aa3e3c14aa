// soft_mul.cuh -- FP64 products on the integer pipe, the bits of a * b.
//
// GB300 issues an FP64 instruction in 64 to 78 cycles of an SM sub-partition and,
// beside it, up to 32 multiply-adds of 32-bit words. A correctly rounded
// product takes about 40 integer instructions, four of them multiplies: a
// kernel bound by the FP64 pipe gains where it moves some products over.
//
// The significands, left-aligned in 64 bits, are multiplied to 128 bits; the
// upper 64, the lowest bit set if anything below is, are normalised and rounded
// to nearest even. Zeros give zeros. Where an operand is subnormal, infinite or
// NaN, or the result would not be normal, *ok turns false and the value
// returned means nothing.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define TFS_SOFT __host__ __device__ __forceinline__
#else
#define TFS_SOFT inline
#endif

namespace tfs {
namespace soft {

struct Words {
  unsigned lo, hi;
};

TFS_SOFT Words words(double x) {
#if defined(__CUDA_ARCH__)
  return {(unsigned)__double2loint(x), (unsigned)__double2hiint(x)};
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return {(unsigned)u, (unsigned)(u >> 32)};
#endif
}

TFS_SOFT double value(unsigned lo, unsigned hi) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

// a * b + c
TFS_SOFT uint64_t mad_wide(unsigned a, unsigned b, uint64_t c) {
#if defined(__CUDA_ARCH__)
  uint64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (uint64_t)a * b + c;
#endif
}

// {hi, lo} << s, the upper word (s < 32)
TFS_SOFT unsigned shl(unsigned lo, unsigned hi, unsigned s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return s == 0 ? hi : (hi << s) | (lo >> (32 - s));
#endif
}

// {hi, lo} >> s, the lower word (0 < s < 32)
TFS_SOFT unsigned shr(unsigned lo, unsigned hi, unsigned s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return (hi << (32 - s)) | (lo >> s);
#endif
}

TFS_SOFT double mul(double a, double b, bool *ok) {
  const Words u = words(a), v = words(b);
  const unsigned ea = (u.hi >> 20) & 0x7ffu, eb = (v.hi >> 20) & 0x7ffu;
  const bool za = ((u.hi << 1) | u.lo) == 0u, zb = ((v.hi << 1) | v.lo) == 0u;
  // significands, the leading bit at bit 63
  const unsigned ah = 0x80000000u | (shl(u.lo, u.hi, 11) & 0x7fffffffu), al = u.lo << 11;
  const unsigned bh = 0x80000000u | (shl(v.lo, v.hi, 11) & 0x7fffffffu), bl = v.lo << 11;
  const uint64_t p0 = mad_wide(al, bl, 0);
  const uint64_t p1 = mad_wide(al, bh, p0 >> 32);
  const uint64_t p2 = mad_wide(ah, bl, (unsigned)p1);
  const uint64_t p3 = mad_wide(ah, bh, p1 >> 32) + (p2 >> 32);
  const unsigned h = (unsigned)(p3 >> 32), l = (unsigned)p3, low = (unsigned)p2;
  // leading bit at 63 (carry) or 62 of the upper 64
  const unsigned carry = h >> 31, s = 1u - carry;
  const unsigned nh = shl(l, h, s);
  const unsigned nl = shl(low, l, s) | ((low | (unsigned)p0) != 0u ? 1u : 0u);
  // 53 bits, and the 11 below them
  const unsigned ql = shr(nl, nh, 11), qh = nh >> 11;
  const unsigned up = (nl & 0x7ffu) + (ql & 1u) > 0x400u ? 1u : 0u;
  const unsigned e = ea + eb + carry - 1023u;  // of the result, before a rounding carry
  const uint64_t r = ((uint64_t)((e - 1u) << 20) << 32) + (((uint64_t)qh << 32) | ql) + up;
  const unsigned sign = (u.hi ^ v.hi) & 0x80000000u;
  const bool zero = za || zb;
  // both normal, and 1 <= e <= 2045 (2046 might round up to infinity)
  const bool fine = ea - 1u < 2046u && eb - 1u < 2046u && e - 1u < 2045u;
  *ok = *ok && (fine || (za && eb < 2047u) || (zb && ea < 2047u));
  return value(zero ? 0u : (unsigned)r, sign | (zero ? 0u : (unsigned)(r >> 32)));
}

}  // namespace soft
}  // namespace tfs
