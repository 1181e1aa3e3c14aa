// fx_pair.cuh -- the far-field RPY pair in 64-bit fixed point.
//
// Why. On this GPU one FP64 warp instruction holds an SM sub-partition's FP64
// pipe for 78 cycles, a 32 x 32 + 64-bit integer multiply-add (IMAD.WIDE) for
// two (measured with chains of each over every SM). A value kept as a 64-bit
// integer of known scale multiplies in three IMAD.WIDE (the two high-by-low
// products and the high one; the low-by-low product is below the last place),
// so the pair costs about an eighth of its FP64 form, and its absolute error
// is smaller: sums of 62-bit products kept exact in 96-bit accumulators
// against FP64's 53 bits at every addition.
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
// below 0.74 (a_i + a_j) (fx_lx): with r > a_i + a_j every power of lambda/r
// and every coefficient below stays under 1. Positions are round((x - o)
// 2^(61 - Ex)), |x - o| < 2^Ex (FxFrame), forces round(F 2^(61 - es)) with
// |F| <= 2^es and |T| <= lambda 2^es over the chunk of sources.
//
// The pair, with w = d/r up to the FP32 seed's error, kappa = 1/|w|^2 and
// lambda = 1 (d = x_i - x_j, units of 1/(8 pi mu)):
//   v_t += A F + c w + (rho T) x w      A = (1 + s/r^2)/r, rho = kappa^(1/2)/r^2
//   v_r += (rho F) x w - T/(2 r^3) + q w
//   c = kappa (1 - 3 s/r^2)/r (w.F),  q = 3 kappa/(2 r^3) (w.T)
// (the far field of cuda_functions.cu:224-316). The reciprocal square root is
// the FP32 hardware estimate y of 1/|d|, corrected by its own residual
// e = 1 - |w|^2, w = d y, which is exact to the last place: 1/|d| =
// y (1 + e/2 + 3 e^2/8) and kappa = 1 + e + e^2 (binomial series; |e| < 2^-19
// leaves terms below 2^-57).
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
TFS_FX Limb negatable(u64 pb) {
  const int l = (int)((unsigned)pb ^ 0x80000000u);
  return {(int)(pb >> 32), l > -0x7fffffff ? l : -0x7fffffff};
}
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

// Middle sums start at 2^63, and for a result shifted left by S at 2^(63 - S)
// more, so that after the shift the bias is 2^31 plus 2^(S - 1) high words;
// plus half a unit of the truncation to the high word.
constexpr u64 kHalf = 0x80000000ull;
template <int S>
TFS_FX constexpr u64 mid0() {
  return (1ull << 63) + (S > 0 ? 1ull << (63 - S) : 0ull) + 0x80000000ull;
}
TFS_FX u64 mid_add(u64 m, Limb a, Limb b) { return madw(a.l, b.h, madw(a.h, b.l, m)); }

// a b 2^S: unit 2^-(fa + fb - 64 + S)
template <int S>
TFS_FX Limb mul(Limb a, Limb b) {
  const u64 p = madw(a.h, b.h, mid_add(mid0<S>(), a, b) >> 32);
  if (S == 0) return limb(p);
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

// Sum of many products: 128 bits, unsigned; the middle sums' low words are
// kept. Every addend carries the bias 2^62 + 2^31 in its high 96 bits (not
// negative, so no sign extension); the reader takes it off.
struct Acc {
  unsigned w0, w1, w2, w3;
};
constexpr u64 kAccHigh0 = 1ull << 62, kAccMid0 = 1ull << 63;  // starts of an addend's sums
// += high products, with the middle sum m (p: high products + m's high word)
TFS_FX void acc_add(Acc &a, u64 p, u64 m) {
#ifdef __CUDA_ARCH__
  asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\t"
      "addc.u32 %3, %3, 0;"
      : "+r"(a.w0), "+r"(a.w1), "+r"(a.w2), "+r"(a.w3)
      : "r"(low(m)), "r"(low(p)), "r"(high(p)));
#else
  u64 s = (u64)a.w0 + low(m);
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

// Add the pair to v[0..2] (VD = 6: and v[3..5]); sums of the unit 2^-59. x,
// xs: target and source position words; f, t: force and torque (FD = 6),
// 2^-62. Returns whether the pair is at or inside contact: it then adds its
// biases only.
template <int VD, int FD>
TFS_FX bool far_pair(Acc *v, const u64 *x, const u64 *xs, const Limb *f, const Limb *t,
                     const PairFx &pc) {
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
  Limb w[3];  // d y: 2^-62, |w| <= 1 + 2^-19
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
  const Limb kappa = {(int)(high(km) + (low(km) >> 31)) + (1 << 28), (int)low(km)};  // 2^-60
  // 1 + e/2 + 3 e^2/8: 2^-62
  const u64 g = km + e + ((1ull << 62) + (e2 >> 1));
  // lambda/r: 2^-63, below 0.74
  const u64 g2 = g << 1;
  const u64 r = umadw(Y << 1, high(g2), umadw(Y << 1, low(g2), 0ull) >> 32);
  const unsigned nr = nw + (unsigned)pc.shift - 30u;  // 0 .. 11
  const Limb r1 = limb2(funnel_r(low(r), high(r), nr), funnel_r(high(r), 0u, nr));
  const Limb r2 = mul<0>(r1, r1);  // 1/r^2: 2^-62, below 0.55
  // s/r^2, at most 1/3, plus 2^31 (and 2^2 high words): 2^-62
  const u64 sp = madw(pc.s.h, r2.h, mid_add(mid0<3>(), pc.s, r2) >> 32) << 3;
  const Limb al = limb(sp + ((1ull << 62) - (4ull << 32)));  // 1 + s/r^2
  const Limb be =
      limb((1ull << 62) + (12ull << 32) + 4ull * 0x80000000ull - 3ull * sp);  // 1 - 3 s/r^2
  const Limb A = mul<0>(r1, al);             // 2^-61, below 0.99
  const Limb rk = mul<0>(r1, kappa);         // kappa/r: 2^-59
  const Limb B = mul<6>(rk, be);             // kappa (1 - 3 s/r^2)/r: 2^-63, below 0.74
  const Limb c = mul<2>(B, dot(w, f));       // (w.F: 2^-60) 2^-61, below 0.74
  Limb xr[3], xm[3], h, p;  // rho w and its negative, -1/(2 r^3) and q: 2^-61
  if (FD == 6 || VD == 6) {
    const Limb rho = mul<3>(r2, limb(g + 0x80000000ull));  // 2^-63, below 0.55
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 3; ++k) {
      xr[k] = negatable(madw(rho.h, w[k].h, mid_add(mid0<0>(), rho, w[k]) >> 32));
      xm[k] = minus(xr[k]);
    }
    if (FD == 6 && VD == 6) {
      // 1/r^3: 2^-61; a bias of any of the three would add up over sources with
      // like torques
      const u64 r3 = madw(r2.h, r1.h, mid_add(mid0<0>(), r2, r1) >> 32) - 0x80000000ull;
      h = minus(negatable(((r3 + 1ull) >> 1) + 0x80000000ull));
      // 3/(2 r^3): 2^-63, below 0.61
      p = mul<2>(mul<4>(limb(6ull * r3 + 0x80000000ull), kappa), dot(w, t));
    }
  }
  // every addend's middle sums add 2^31 each to its bias
  const u64 high0 = FD == 6 ? kAccHigh0 - kHalf : kAccHigh0;
  // four middle terms to a sum, each at most 2^61, and (h, p) smaller
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 0; k < 3; ++k) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    u64 m1 = mid_add(mid_add(kAccMid0, A, f[k]), c, w[k]);
    u64 hh = madw(A.h, f[k].h, madw(c.h, w[k].h, high0 + (m1 >> 32)));
    if (FD == 6) {  // (rho T) x w
      const u64 m2 = mid_add(mid_add(mid0<0>(), t[a], xr[b]), t[b], xm[a]);
      hh = madw(t[a].h, xr[b].h, madw(t[b].h, xm[a].h, hh + (m2 >> 32)));
    }
    acc_add(v[k], hh, m1);
    if (VD == 6) {  // (rho F) x w
      m1 = mid_add(mid_add(kAccMid0, f[a], xr[b]), f[b], xm[a]);
      hh = madw(f[a].h, xr[b].h, madw(f[b].h, xm[a].h, high0 + (m1 >> 32)));
      if (FD == 6) {
        const u64 m2 = mid_add(mid_add(mid0<0>(), h, t[k]), p, w[k]);
        hh = madw(h.h, t[k].h, madw(p.h, w[k].h, hh + (m2 >> 32)));
      }
      acc_add(v[3 + k], hh, m1);
    }
  }
  return near;
}

}  // namespace fx
}  // namespace tfs
