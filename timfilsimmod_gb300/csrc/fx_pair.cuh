// fx_pair.cuh -- the far-field RPY pair in 64-bit fixed point.
//
// Why. On this GPU one FP64 warp instruction holds an SM sub-partition's FP64
// pipe for 78 cycles, a 32 x 32 + 64-bit integer multiply-add (IMAD.WIDE) for
// two (measured with chains of each over every SM). A value kept as a 64-bit
// integer of known scale multiplies in three IMAD.WIDE (the two high-by-low
// products and the high one; the low-by-low product is below the last place),
// so the pair costs about a seventh of its FP64 form, and its errors are smaller:
// 59 to 62 places against FP64's 53, sums kept exact in 128-bit accumulators.
//
// Values. A value v is held as the integer round(v 2^f), split into a signed
// high word and a signed low word (Limb); f is a property of the variable,
// written in its comment as "2^-f". A product of limbs a (2^-fa) and b (2^-fb)
// has the unit 2^-(fa + fb - 64). The middle sum of a product carries the bias
// 2^63, so that it is not negative and its high word can be added without a
// sign extension; the bias leaves 2^31 in the result, which is the rounding
// constant of its split into limbs: the split then costs one addition. Two
// middle terms are at most 2^61 each in magnitude times the operands' sizes;
// every sum below stays under 2^63 with the sizes written beside it.
//
// Scales. Lengths are measured in lambda = 2^lx, the largest power of two
// below 0.74 (a_i + a_j) (fx_lambda_exponent): lambda/r and s/r^2 stay under 1. Positions
// are round((x - o) 2^(61 - Ex)), |x - o| < 2^Ex (frame_of); a source's force
// and torque are round(F 2^(62 - es + below)), |F| <= 2^(es - below), |T| <=
// lambda 2^(es - below), es the exponent of the job's largest.
//
// Relative accuracy. Every power of 1/r is held as a number in [1/8, 1) times a
// power of two: lambda/r = a 2^-n, a in [1/2, 1), and coefficients are formed
// of a alone, so they have their 59 to 62 places whatever the distance. A
// pair's terms are shifted into place as whole sums: the torque's by n against
// the force's, all by n (v_t) or 2 n (v_r), and by the source's below, into
// 128-bit sums whose last place is 2^-91 of the largest force over lambda. The
// 2-norm error of each of the four couplings (force or torque to velocity or
// angular velocity) is below 2^-51 of its own size from contact to 1000 radii
// (tests/test_fixed_pair_relative.py). (With coefficients held to a fixed place,
// 2^-61, the angular velocity of a torque was off by 3e-13 of itself at 50 radii and
// 5e-11 at 300, that of a force by 2e-15 and 6e-14.)
//
// The pair, with w = d/r up to the FP32 seed's error, kappa = 1/|w|^2 and
// lambda = 1 (d = x_i - x_j, units of 1/(8 pi mu)):
//   v_t += A F + c w + (rho T) x w      A = (1 + s/r^2)/r, rho = kappa^(1/2)/r^2
//   v_r += (rho F) x w - T/(2 r^3) + q w
//   c = kappa (1 - 3 s/r^2)/r (w.F),  q = 3 kappa/(2 r^3) (w.T)
// where the code has a in place of 1/r and shifts the sums
// (the far field of cuda_functions.cu:224-316). The reciprocal square root is
// the FP32 hardware estimate y of 1/|d|, corrected by its own residual
// e = 1 - |w|^2, w = d y, which is exact to the last place: 1/|d| =
// y (1 + e/2 + 3 e^2/8) and kappa = 1 + e + e^2 (binomial series; |e| < 2^-18.4,
// most of it from the FP32 separation at contact in the widest frame, leaves
// terms below 2^-55).
//
// The same source compiles for the host (tests/test_fixed_pair.py checks it
// there against quadruple precision).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define TFS_FX __host__ __device__ __forceinline__
#else
#define TFS_FX inline
#endif

namespace tfs {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

struct Limb {
  int h, l;  // h 2^32 + l, both signed
};

// P + 2^31 -> limbs of P
TFS_FX Limb limb(u64 pb) { return {(int)(pb >> 32), (int)((unsigned)pb + 0x80000000u)}; }
// words of P -> limbs of P
TFS_FX Limb limb2(unsigned lo, unsigned hi) { return {(int)(hi + (lo >> 31)), (int)lo}; }
TFS_FX Limb limb_of(i64 v) { return limb((u64)v + 0x80000000ull); }
// Limbs that can be negated: the low word is not -2^31 (one place off where it
// would be). Zero stays zero.
TFS_FX Limb negatable(Limb a) { return {a.h, a.l > -0x7fffffff ? a.l : -0x7fffffff}; }
TFS_FX Limb minus(Limb a) { return {-a.h, -a.l}; }

// a b + c: one IMAD.WIDE
TFS_FX u64 madw(int a, int b, u64 c) {
#ifdef __CUDA_ARCH__
  u64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (u64)((i64)a * (i64)b) + c;
#endif
}
TFS_FX u64 umadw(unsigned a, unsigned b, u64 c) {
#ifdef __CUDA_ARCH__
  u64 d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (u64)a * (u64)b + c;
#endif
}
TFS_FX unsigned low(u64 v) { return (unsigned)v; }
TFS_FX unsigned high(u64 v) { return (unsigned)(v >> 32); }
TFS_FX u64 pack64(unsigned lo, unsigned hi) { return ((u64)hi << 32) | lo; }
// the low word of (hi:lo) >> n and the high word of (hi:lo) << n, n in [0, 31]
TFS_FX unsigned funnel_r(unsigned lo, unsigned hi, unsigned n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, n);
#else
  return (unsigned)(pack64(lo, hi) >> (n & 31u));
#endif
}
TFS_FX unsigned funnel_l(unsigned lo, unsigned hi, unsigned n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, n);
#else
  return (unsigned)((pack64(lo, hi) << (n & 31u)) >> 32);
#endif
}

// Middle sums start at 2^63, and for a result shifted left by S > 1 at 2^(63 - S)
// more, so that after the shift the bias is 2^31 plus 2^(S - 1) high words;
// plus half a unit of the truncation to the high word. (S = 1 has no room for
// that beside two middle terms of 2^61: its bias is taken off before.)
constexpr u64 kHalf = 0x80000000ull;
template <int S>
TFS_FX constexpr u64 mid0() {
  return (1ull << 63) + (S > 1 ? 1ull << (63 - S) : 0ull) + kHalf;
}
TFS_FX u64 mid_add(u64 m, Limb a, Limb b) { return madw(a.l, b.h, madw(a.h, b.l, m)); }

// a b 2^S: unit 2^-(fa + fb - 64 + S)
template <int S>
TFS_FX Limb mul(Limb a, Limb b) {
  const u64 p = madw(a.h, b.h, mid_add(mid0<S>(), a, b) >> 32);
  if (S == 0) return limb(p);
  if (S == 1) return limb2(low(p) << 1, funnel_l(low(p), high(p), 1) - 1u);
  return {(int)funnel_l(low(p), high(p), S) - (1 << (S > 0 ? S - 1 : 0)),
          (int)((low(p) << S) + 0x80000000u)};
}
// a . b
TFS_FX Limb dot(const Limb *a, const Limb *b) {
  const u64 m = mid_add(mid_add(mid_add(mid0<0>(), a[0], b[0]), a[1], b[1]), a[2], b[2]);
  return limb(madw(a[0].h, b[0].h, madw(a[1].h, b[1].h, madw(a[2].h, b[2].h, m >> 32))));
}

TFS_FX float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (float)(1.0 / sqrt((double)x));
#endif
}
TFS_FX unsigned float_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  unsigned u;
  memcpy(&u, &x, 4);
  return u;
#endif
}

// A term of 96 bits, signed: a sum of high products p over the low word of its
// middle sum m.
struct Term {
  unsigned lo, mid, hi;
};
TFS_FX Term term(u64 p, u64 m) { return {low(m), low(p), high(p)}; }
TFS_FX u64 high_signed(u64 m) { return (u64)((i64)m >> 32); }
// >> n, n in [0, 31]
TFS_FX Term shr(Term t, unsigned n) {
  return {funnel_r(t.lo, t.mid, n), funnel_r(t.mid, t.hi, n), (unsigned)((int)t.hi >> n)};
}
TFS_FX Term add(Term a, Term b) {
#ifdef __CUDA_ARCH__
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(a.lo), "+r"(a.mid), "+r"(a.hi)
      : "r"(b.lo), "r"(b.mid), "r"(b.hi));
  return a;
#else
  u64 s = (u64)a.lo + b.lo;
  const unsigned l = low(s);
  s = (u64)a.mid + b.mid + (s >> 32);
  return {l, low(s), a.hi + b.hi + high(s)};
#endif
}

// Sum of many terms: 128 bits. Every addend carries the bias 2^62 + 2^31 in its
// upper 64 bits (not negative, so no sign extension); the reader takes it off.
struct Acc {
  unsigned w0, w1, w2, w3;
};
TFS_FX void acc_add(Acc &a, Term t) {
  const u64 p = pack64(t.mid, t.hi) + ((1ull << 62) + kHalf);
#ifdef __CUDA_ARCH__
  asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\t"
      "addc.u32 %3, %3, 0;"
      : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2), "+r"(a.w3)
      : "r"(t.lo), "r"(low(p)), "r"(high(p)));
#else
  u64 s = (u64)a.w0 + t.lo;
  a.w0 = low(s);
  s = (u64)a.w1 + low(p) + (s >> 32);
  a.w1 = low(s);
  s = (u64)a.w2 + high(p) + (s >> 32);
  a.w2 = low(s);
  a.w3 += high(s);
#endif
}

// Per (target kind, source kind) constants of a launch.
struct PairFx {
  float near_q;  // (a_i + a_j)^2 2^(58 - 2 Ex), widened: r^2 at or below it is left out
  int shift;     // Ex - lx, 1 .. 10
  Limb s;        // (a_i^2 + a_j^2)/(3 lambda^2), below 3.9: 2^-61
};
constexpr int kMaxShift = 10;
constexpr unsigned kMaxBelow = 9;  // 2 n + below <= 31, n <= kMaxShift + 1

// Add the pair to v[0..2] (VD = 6: and v[3..5]); sums of the unit 2^-59 (and
// 32 places below). x, xs: target and source position words; f, t: force and
// torque (FD = 6), 2^-62, times 2^-below (at most kMaxBelow). Returns whether
// the pair is at or inside contact: it then adds its biases only.
template <int VD, int FD>
TFS_FX bool far_pair(Acc *v, const u64 *x, const u64 *xs, const Limb *f, const Limb *t,
                     const PairFx &pc, unsigned below = 0u) {
  u64 d[3];  // 2^-(61 - Ex), |d| < 2^62
  float df[3];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 0; k < 3; ++k) {
    d[k] = x[k] - xs[k];
    df[k] = (float)(int)high(d[k]) + 0.5f;
  }
  const float q = fmaf(df[0], df[0], fmaf(df[1], df[1], df[2] * df[2]));  // r^2 2^(58 - 2 Ex)
  const bool near = !(q > pc.near_q);
  const unsigned yb = float_bits(rsqrt_seed(q));
  // y = Y 2^(-nw - 30), Y in [2^30, 2^31); Y = 0 leaves the pair out
  const unsigned Y = near ? 0u : ((yb << 7) & 0x3fffffffu) | 0x40000000u;
  const unsigned nw = 127u - (yb >> 23);  // 18 .. 31
  Limb w[3];  // d y: 2^-62, |w| <= 1 + 2^-18
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 0; k < 3; ++k) {
    const u64 lo = umadw(low(d[k]), Y, 0ull);
    const u64 hi = madw((int)high(d[k]), (int)Y, lo >> 32);
    w[k] = limb2(funnel_r(low(lo), low(hi), nw), funnel_r(low(hi), high(hi), nw));
  }
  // e = 1 - |w|^2: 2^-60, below 2^42 (the middle sum, below 2^62, counts twice)
  u64 m = madw(w[0].h, w[0].l,
               madw(w[1].h, w[1].l, madw(w[2].h, w[2].l, (1ull << 62) + (1ull << 30))));
  m += m;
  const u64 ww =
      madw(w[0].h, w[0].h, madw(w[1].h, w[1].h, madw(w[2].h, w[2].h, m >> 32)));
  const u64 e = (1ull << 60) + (1ull << 31) - ww;
  const int e14 = (int)funnel_r(low(e), high(e), 14);  // 2^-46
  const unsigned e2 = high(madw(e14, e14, 0ull));      // e^2: 2^-60
  const u64 km = e + e2;                               // kappa - 1
  const Limb kappa = limb((km << 2) + ((1ull << 62) + 0x80000000ull));  // 2^-62
  // 1 + e/2 + 3 e^2/8: 2^-62
  const u64 g = km + e + ((1ull << 62) + (e2 >> 1));
  // lambda/r = a 2^-n: a in [1/2, 1] (up to the seed's error; below 0.74 with n = 0), 2^-62
  const u64 r = umadw(Y << 1, high(g), umadw(Y << 1, low(g), 0ull) >> 32);
  const unsigned n = (nw + (unsigned)pc.shift - 30u) & 31u;  // 0 .. 11
  const unsigned n2 = (2u * n) & 31u;
  const Limb a1 = limb2(low(r), high(r));
  // a^2: 2^-62
  const u64 r2 = (madw(a1.h, a1.h, mid_add(mid0<0>(), a1, a1) >> 32) - kHalf) << 2;
  const Limb a2 = limb2(low(r2), high(r2));
  // 1/r^2, below 0.55: 2^-62
  const Limb s2 = limb2(funnel_r(low(r2), high(r2), n2), high(r2) >> n2);
  // s/r^2, at most 1/3, plus 2^31 (and 2^2 high words): 2^-62
  const u64 sp = madw(pc.s.h, s2.h, mid_add(mid0<3>(), pc.s, s2) >> 32) << 3;
  const Limb al = limb(sp + ((1ull << 62) - (4ull << 32)));  // 1 + s/r^2
  const Limb be =
      limb((1ull << 62) + (12ull << 32) + 4ull * 0x80000000ull - 3ull * sp);  // 1 - 3 s/r^2
  const Limb A = mul<1>(a1, al);                     // 2^-61, below 1.34
  const Limb B = mul<2>(mul<2>(a1, kappa), be);      // a kappa (1 - 3 s/r^2): 2^-62
  const Limb c = mul<3>(B, dot(w, f));               // (w.F: 2^-60) 2^-61, at most 1
  Limb xr[3], xm[3], h, p;  // rho w and its negative, -a^3/2 and q: 2^-61
  if (FD == 6 || VD == 6) {
    const Limb rho = mul<2>(a2, limb(g + 0x80000000ull));  // 2^-62
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 3; ++k) {
      xr[k] = negatable(mul<1>(rho, w[k]));
      xm[k] = minus(xr[k]);
    }
    if (FD == 6 && VD == 6) {
      // a^3, plus 2^31: 2^-60
      const u64 r3 = madw(a2.h, a1.h, mid_add(mid0<0>(), a2, a1) >> 32);
      h = minus(negatable(limb(r3)));
      p = mul<3>(mul<3>(limb(3ull * r3 - 2ull * kHalf), kappa), dot(w, t));
    }
  }
  // four middle terms to a sum, signed, below 2^63
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 0; k < 3; ++k) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    u64 m1 = mid_add(mid_add(0ull, A, f[k]), c, w[k]);
    Term s = term(madw(A.h, f[k].h, madw(c.h, w[k].h, high_signed(m1))), m1);
    if (FD == 6) {  // (rho T) x w
      m1 = mid_add(mid_add(0ull, t[a], xr[b]), t[b], xm[a]);
      s = add(s, shr(term(madw(t[a].h, xr[b].h, madw(t[b].h, xm[a].h, high_signed(m1))), m1),
                     n));
    }
    acc_add(v[k], shr(s, (n + below) & 31u));
    if (VD == 6) {  // (rho F) x w
      m1 = mid_add(mid_add(0ull, f[a], xr[b]), f[b], xm[a]);
      s = term(madw(f[a].h, xr[b].h, madw(f[b].h, xm[a].h, high_signed(m1))), m1);
      if (FD == 6) {
        m1 = mid_add(mid_add(0ull, h, t[k]), p, w[k]);
        s = add(s, shr(term(madw(h.h, t[k].h, madw(p.h, w[k].h, high_signed(m1))), m1), n));
      }
      acc_add(v[3 + k], shr(s, (n2 + below) & 31u));
    }
  }
  return near;
}

}  // namespace fx
}  // namespace tfs
