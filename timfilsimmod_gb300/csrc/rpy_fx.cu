// rpy_fx.cu -- the FP64 work-queue products, with the far-field pairs in
// 64-bit fixed point (fx_pair.cuh).
//
// A product of FP64 jobs runs as two launches: fx_pack_kernel packs the FP64
// records, turns them into fixed-point ones and finds the scales; rpy_fx_kernel
// computes the products. A job whose data the fixed-point form cannot take
// (fx_pack_kernel's verdict, on the device: a swimmer more than 2^10 lambda
// across, forces or positions that are not finite or outside 2^(+-kFxExponent),
// positions outside the frame the origin kernel last saw; or radii too far
// apart for one lambda, known on the host) runs on the FP64 pipe instead, as
// units of rpy_queue.cuh in the same launch.
//
// rpy_fx_kernel. Work units, persistent CTAs, arrival counters and the
// determinism argument are rpy_queue.cuh's. A fixed-point unit's chunk is a
// run of tiles of 32 sources; the chunk sums are kept as 128-bit integers of one
// scale per job, so the last unit of a target block adds the chunks exactly
// and converts once to FP64. Pairs at or inside contact (itself, touching or
// overlapping particles), which the fixed-point pair leaves out and reports
// in a 32-bit mask per tile, are evaluated by the exact three-regime FP64
// formula from the FP64 records and added to the integer sums, rounded to
// their unit.
//
// Bound: issue of the integer multiply-adds (IMAD.WIDE, two cycles each) and
// of the carry additions and shifts between them: some 970 cycles a 6x6 pair,
// warp and SM sub-partition, against 52 FP64 instructions of 78 cycles.
// Occupancy does not matter (3 and 4 CTAs of 128 an SM within 2%).
// Medium swimmer (12 800 segments, 2 562 blobs), FP64 sums and these: M_ss 9.19
// and 4.30 ms, M_bs 1.38 and 0.79, M_sb 1.38 and 0.60, M_bb 0.36 and 0.11. (M_ss
// 3.72, M_bs 0.56, M_sb 0.51 ms with coefficients of a fixed place, whose error
// grows with the distance: fx_pair.cuh.) The error against 64-bit sums is not
// larger, neither in the 2-norm over all velocities (1.5e-15 against 1.9e-15,
// both with the 64-bit sums' own) nor for a target alone, far from the loaded
// particles or with forces far below the largest.
#include <algorithm>
#include <atomic>
#include <cmath>

#include <cuda_runtime.h>

#include "fx_pair.cuh"
#include "rpy_queue.cuh"
#include "rpy_tile.cuh"
#include "tfs_kernels.h"

namespace tfs {

namespace {

using fx::Acc;
using fx::i64;
using fx::Limb;
using fx::u64;

constexpr int kFxPackThreads = 256;
constexpr int kNoForce = kFxEmpty;
// Forces up to 2^(+-kFxExponent) and lambda up to 2^(+-kFxLambda): an exponent es of
// a force, or of a torque over lambda, is then within kFxExponent + kFxLambda + 1, and
// the results' factor 2^(es - 91 - 2 lx) within 2^(+-1000). Beyond, FP64 sums.
constexpr int kFxExponent = 800, kFxLambda = 20;
static_assert(kFxExponent + 3 * kFxLambda + 1 + 91 <= 1000, "pow2's range");

// The frame of a product: positions relative to o in units of 2^(Ex - 61).
struct Frame {
  double o[3];
  int Ex;
  bool ok;
};

// The exponent e with |v| < 2^e of a finite v (not subnormal).
__device__ __forceinline__ int exponent_of(double v) {
  return ((__double2hiint(v) >> 20) & 0x7ff) - 1022;
}

// From the origin kernel's result (centre of the bounds, and a bound of every
// |x_k - o_k|). A swimmer whose bounds hold the coordinates' zero keeps it as
// its origin, so that its positions enter without a rounding.
__device__ Frame frame_of(const double *origin, int lx_min, int lx_max) {
  Frame f;
  double E = 0.0;
  const double ext = origin[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const bool at_zero = fabs(origin[k]) <= ext;
    f.o[k] = at_zero ? 0.0 : origin[k];
    E = fmax(E, at_zero ? ext + fabs(origin[k]) : ext);
  }
  f.ok = E < 1e200 && E >= 0.0;
  int ex = lx_max + 1;
  if (f.ok && E > 0.0) {
    const int e = exponent_of(1.7320509 * E);  // |x - o| < 2^e: r^2 < 2^(2 e + 2)
    ex = e > ex ? e : ex;
  }
  f.Ex = ex;
  f.ok = f.ok && ex - lx_min <= fx::kMaxShift;
  return f;
}

__device__ __forceinline__ double pow2(int e) {  // |e| <= 1000
  return __hiloint2double((e + 1023) << 20, 0);
}

// round(v 2^e) for |v 2^e| < 2^63, by integer shifts: an FP64 multiplication
// and a conversion hold the FP64 pipe longer. v is finite; subnormals read 0.
__device__ __forceinline__ i64 to_fixed(double v, int e) {
  const u64 b = (u64)__double_as_longlong(v);
  const int ev = (int)(b >> 52) & 0x7ff;
  const int s = ev - 1075 + e;
  u64 m = ev == 0 ? 0ull : (b & 0xfffffffffffffull) | (1ull << 52);
  if (s >= 0)
    m <<= s;
  else
    m = s < -60 ? 0ull : (m + (1ull << (-s - 1))) >> -s;
  return (i64)b < 0 ? -(i64)m : (i64)m;
}

// One thread per source of the two record arrays (segments first, each array
// padded to whole warps): fixed-point records, each source's force with an
// exponent of its own (and, from plain arrays, the FP64 records, which saves two
// launches a product); the last CTA writes the sets' exponents and the verdict.
// Latency bound; 45 FP64 instructions a thread made it 7.3 us, integer shifts
// and FP32 norms in their place 7.1 us (4 876 particles): the atomics' round trips.
__global__ void __launch_bounds__(kFxPackThreads) fx_pack_kernel(const FxSystem q) {
  __shared__ int s_bad, s_es[2];
  __shared__ bool s_last;
  __shared__ Frame s_fr;
  if (threadIdx.x == 0) {
    s_bad = 0;
    s_es[0] = s_es[1] = kNoForce;
    s_fr = frame_of(q.origin, q.lx_min, q.lx_max);
  }
  const int tiles_s = (q.n[0] + 31) / 32;
  const int tile = (blockIdx.x * kFxPackThreads + threadIdx.x) / 32, lane = threadIdx.x & 31;
  const int set = tile < tiles_s ? 0 : 1;
  const int local = set == 0 ? tile : tile - tiles_s;
  const int i = local * 32 + lane;
  const int fd = q.fd[set], len = fd == 6 ? 10 : 6;
  const bool warp_in = local * 32 < q.n[set], in = i < q.n[set];
  double f[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, x[3] = {0.0, 0.0, 0.0};
  if (in) {
    double *r = q.rec[set] + (size_t)i * len;
    const bool raw = q.x[set] != nullptr;
    const double *px = raw ? q.x[set] + 3 * (size_t)i : r;
    const double *pf = raw ? q.f[set] + (size_t)fd * i : r + 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x[k] = px[k];
      f[k] = pf[k];
      if (fd == 6) f[3 + k] = pf[3 + k];
    }
    if (raw) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        r[k] = x[k];
        r[3 + k] = f[k];
        if (fd == 6) r[6 + k] = f[3 + k];
      }
      if (fd == 6) r[9] = 0.0;
    }
  }
  __syncthreads();
  const Frame fr = s_fr;
  if (warp_in) {  // whole warps
    bool bad = !fr.ok;
    const double reach = bad ? 0.0 : pow2(fr.Ex) * 0.57735;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (fr.o[k] != 0.0) x[k] -= fr.o[k];
      bad = bad || !(fabs(x[k]) <= reach);
    }
    int e = kNoForce;
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // |F| < 2^e, |T| < 2^(e + lx_min)
      int e0 = kNoForce;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double v = f[3 * h + k];
        if (v != 0.0) e0 = max(e0, exponent_of(v));
      }
      if (e0 > kNoForce) {
        bad = bad || e0 > kFxExponent || e0 < -kFxExponent;  // and infinities, NaN, subnormals
        if (!bad) {
          // the norm of the components over 2^e0, in FP32 (relative error 2^-21)
          float n2 = 0.f;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float c = (float)(int)(to_fixed(f[3 * h + k], 30 - e0)) * 9.31322575e-10f;
            n2 = fmaf(c, c, n2);
          }
          e = max(e, e0 + (n2 >= 0.99999f ? 1 : 0) - (h ? q.lx_min : 0));
        }
      }
    }
    bad = bad && in;
    int top = e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (bad) atomicOr(&s_bad, 1);
    if (lane == 0) atomicMax(&s_es[set], top);
    if (in) q.te[set][i] = e;
    if (in && !bad) {
      i64 *w = q.fx[set] + (size_t)i * (fd == 6 ? 9 : 6);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        w[k] = to_fixed(x[k], 61 - fr.Ex);
        w[3 + k] = to_fixed(f[k], 62 - e);
        if (fd == 6) w[6 + k] = to_fixed(f[3 + k], 62 - e - q.lx_min);
      }
    }
  }
  __syncthreads();
  FxState *st = q.state;
  if (threadIdx.x == 0) {
    if (s_bad) atomicOr(&st->bad, 1);
    atomicMax(&st->es_next[0], s_es[0]);
    atomicMax(&st->es_next[1], s_es[1]);
    __threadfence();
    s_last = atomicAdd(&st->arrived, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (s_last && threadIdx.x < 3) {  // one word a thread: their round trips overlap
    if (threadIdx.x == 0) {
      st->Ex = fr.Ex;
      st->arrived = 0u;
      st->ok = atomicExch(&st->bad, 0) == 0 && fr.ok;
    } else {
      st->es[threadIdx.x - 1] = atomicExch(&st->es_next[threadIdx.x - 1], kNoForce);
    }
  }
}

// The pair at or inside contact, exact, in FP64 (r = 0: the self term).
template <int VD, int FD>
__device__ __noinline__ void exact_pair(double *v, const double *xt, const double *rec,
                                        const double *pc) {
  double f[FD];
  const double dx = xt[0] - rec[0], dy = xt[1] - rec[1], dz = xt[2] - rec[2];
#pragma unroll
  for (int k = 0; k < FD; ++k) f[k] = rec[3 + k];
#pragma unroll
  for (int k = 0; k < VD; ++k) v[k] = 0.0;
  const PairConst<double> c{pc[0], pc[1], pc[2], pc[3], pc[4]};
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  if (r2 == 0.0) {
    // the nested branch of the pair function without its r terms
    const double am = fmax(c.ai, c.aj), A = 4.0 / (3.0 * am);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = A * f[k];
    if (VD == 6 && FD == 6) {
      const double R = 1.0 / (am * am * am);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[VD - 3 + k] = R * f[FD - 3 + k];
    }
    return;
  }
  rpy_pair<double, VD, FD>(v, dx, dy, dz, f, c);
}

__device__ __forceinline__ void add128(unsigned (&a)[4], unsigned b0, unsigned b1, unsigned b2,
                                       unsigned b3) {
  asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\t"
      "addc.u32 %3, %3, %7;"
      : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3])
      : "r"(b0), "r"(b1), "r"(b2), "r"(b3));
}

// a += round(v 2^e), |v 2^e| < 2^95, by integer shifts as to_fixed.
__device__ __forceinline__ void acc_add_fixed(Acc &a, double v, int e) {
  const u64 b = (u64)__double_as_longlong(v);
  const int ev = (int)(b >> 52) & 0x7ff;
  const int s = min(ev - 1075 + e, 63);
  const u64 m = ev == 0 ? 0ull : (b & 0xfffffffffffffull) | (1ull << 52);
  u64 lo = 0ull, hi = 0ull;
  if (s >= 0) {
    lo = m << s;
    hi = s > 0 ? m >> (64 - s) : 0ull;
  } else if (s >= -60) {
    lo = (m + (1ull << (-s - 1))) >> -s;
  }
  if ((i64)b < 0) {
    lo = 0ull - lo;
    hi = ~hi + (lo == 0ull ? 1ull : 0ull);
  }
  unsigned w[4] = {a.w0, a.w1, a.w2, a.w3};
  add128(w, fx::low(lo), fx::high(lo), fx::low(hi), fx::high(hi));
  a.w0 = w[0];
  a.w1 = w[1];
  a.w2 = w[2];
  a.w3 = w[3];
}

constexpr int kFp64Tile = 128;  // sources per staged tile of the FP64 units (fixes their sums' order)

// 16-byte aligned records of a staged source: position words, force limbs,
// torque limbs, the exponent below the job's.
template <int FD>
struct Staged {
  static constexpr int words = FD == 6 ? 20 : 16;  // 32-bit
  static constexpr int below = FD == 6 ? 18 : 12;
};

__device__ __forceinline__ Limb shifted(i64 v, int s) {
  if (s > 0) v = (v + (1ll << (s - 1))) >> s;
  return fx::limb_of(v);
}

// The sources of tiles [t0, t1) of one source set into the unit's sums.
template <int VD, int FD, int BLOCK>
__device__ __forceinline__ void sum_tiles(Acc (&v)[VD], const u64 (&xt)[3], const double *tgt,
                                          const QueueJob &job, int set, int t0, int t1, int es,
                                          int Ex, unsigned *smem, bool active, unsigned &count) {
  constexpr int W = Staged<FD>::words;
  constexpr int TS = 64;  // sources staged at a time
  const FxSource &src = job.fx[set];
  const int n = set == 0 ? job.n_a : job.n_b;
  const double *rec = reinterpret_cast<const double *>(set == 0 ? job.src_a : job.src_b);
  fx::PairFx pc;
  pc.shift = Ex - src.lx;
  pc.s = src.s;
  pc.near_q = src.near_q * __int_as_float((127 + 58 - 2 * pc.shift) << 23);
  const int up = 91 - es + src.lx;  // v -> integer: 2^91 lambda / 2^es
  const int s1 = min(t1 * 32, n);
  for (int base = t0 * 32; base < s1; base += TS) {
    const int cnt = min(TS, s1 - base);
    __syncthreads();
    for (int j = threadIdx.x; j < cnt; j += BLOCK) {
      const i64 *w = src.rec + (size_t)(base + j) * (FD == 6 ? 9 : 6);
      // a source up to 2^kMaxBelow smaller than the job's largest keeps all its
      // places (the pair shifts its sums); below, the places that are lost are
      // 2^-71 of the largest
      const int es_below = es - src.te[base + j];
      const int below = min(es_below, (int)fx::kMaxBelow);
      const int sh = min(es_below - below, 63);
      const int sht = min(sh + src.tshift, 63);
      smem[j * W + Staged<FD>::below] = (unsigned)below;
      u64 *o = reinterpret_cast<u64 *>(smem + j * W);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        o[k] = (u64)w[k];
        const Limb F = shifted(w[3 + k], sh);
        o[3 + k] = fx::pack64((unsigned)F.l, (unsigned)F.h);
        if (FD == 6) {
          const Limb T = shifted(w[6 + k], sht);
          o[6 + k] = fx::pack64((unsigned)T.l, (unsigned)T.h);
        }
      }
    }
    __syncthreads();
    if (!active) continue;
    for (int sub = 0; sub < cnt; sub += 32) {
      const int m = min(32, cnt - sub);
      unsigned near = 0u;
#pragma unroll 1
      for (int j = 0; j < m; ++j) {
        const ulonglong2 *o = reinterpret_cast<const ulonglong2 *>(smem + (sub + j) * W);
        const ulonglong2 a = o[0], b = o[1], c = o[2];
        const u64 xs[3] = {a.x, a.y, b.x};
        Limb f[3], t[3];
        f[0] = {(int)(b.y >> 32), (int)b.y};
        f[1] = {(int)(c.x >> 32), (int)c.x};
        f[2] = {(int)(c.y >> 32), (int)c.y};
        if (FD == 6) {
          const ulonglong2 d = o[3];
          const u64 e = *reinterpret_cast<const u64 *>(o + 4);
          t[0] = {(int)(d.x >> 32), (int)d.x};
          t[1] = {(int)(d.y >> 32), (int)d.y};
          t[2] = {(int)(e >> 32), (int)e};
        }
        const unsigned below = smem[(sub + j) * W + Staged<FD>::below];
        if (fx::far_pair<VD, FD>(v, xt, xs, f, t, pc, below)) near |= 1u << j;
      }
      while (near) {
        const int j = __ffs(near) - 1;
        near &= near - 1;
        double u[VD];
        exact_pair<VD, FD>(u, tgt, rec + (size_t)(base + sub + j) * (FD == 6 ? 10 : 6),
                           job.pc64[set]);
#pragma unroll
        for (int k = 0; k < VD; ++k) acc_add_fixed(v[k], u[k], k < 3 ? up : up + src.lx);
      }
    }
    count += (unsigned)cnt;
  }
}

// A chunk's sum, signed, unit 2^-91.
struct __align__(16) Sum128 {
  unsigned w[4];
};

template <int VD, int FDA, int FDB, int BLOCK>
__device__ __forceinline__ void fx_unit(const QueueJob &job, int blk, int c, unsigned *smem,
                                        int *s_last) {
  const int n_tgt = job.n_tgt;
  const int i0 = blk * BLOCK + threadIdx.x;
  const int i = min(i0, n_tgt - 1);  // duplicate the last target; not written
  const bool active = blk * BLOCK + (int)(threadIdx.x & ~31u) < n_tgt;
  const FxState *st = job.fx_state;
  const int Ex = st->Ex;
  int es = job.n_a > 0 ? st->es[job.fx[0].set] : kNoForce;
  if (FDB > 0 && job.n_b > 0) es = max(es, st->es[job.fx[1].set]);
  es = es == kNoForce ? 0 : es;  // no force at all: zeros
  const double *tgt = reinterpret_cast<const double *>(job.tgt_rec) + (size_t)i * (VD == 6 ? 10 : 6);
  u64 xt[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    xt[k] = (u64)job.fx_tgt[(size_t)i * (VD == 6 ? 9 : 6) + k];
  Acc v[VD];
#pragma unroll
  for (int k = 0; k < VD; ++k) v[k].w0 = v[k].w1 = v[k].w2 = v[k].w3 = 0u;
  unsigned count = 0u;
  const int ta = (job.n_a + 31) / 32, tb = FDB > 0 ? (job.n_b + 31) / 32 : 0;
  const int t0 = c * job.fx_chunk, t1 = min(t0 + job.fx_chunk, ta + tb);
  if (t0 < ta)
    sum_tiles<VD, FDA, BLOCK>(v, xt, tgt, job, 0, t0, min(t1, ta), es, Ex, smem, active, count);
  if constexpr (FDB > 0) {
    if (t1 > ta)
      sum_tiles<VD, FDB, BLOCK>(v, xt, tgt, job, 1, max(t0 - ta, 0), t1 - ta, es, Ex, smem, active,
                                count);
  }
  // the sums without their biases
  Sum128 sum[VD];
#pragma unroll
  for (int k = 0; k < VD; ++k) {
    // count (2^62 + 2^31) off the upper 96 bits
    const u64 b0 = (u64)count << 31, b1 = ((u64)count << 62) + b0;
    const unsigned top = (unsigned)(count >> 2) + (b1 < b0 ? 1u : 0u);
    u64 lo = fx::pack64(v[k].w1, v[k].w2);
    const u64 l = lo - b1;
    sum[k].w[0] = v[k].w0;
    sum[k].w[1] = (unsigned)l;
    sum[k].w[2] = (unsigned)(l >> 32);
    sum[k].w[3] = v[k].w3 - top - (lo < b1 ? 1u : 0u);
  }
  if (job.fx_chunks > 1) {
    uint4 *p = reinterpret_cast<uint4 *>(job.partial);
    if (i0 < n_tgt) {
#pragma unroll
      for (int k = 0; k < VD; ++k)
        p[((size_t)c * VD + k) * n_tgt + i0] =
            make_uint4(sum[k].w[0], sum[k].w[1], sum[k].w[2], sum[k].w[3]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      *s_last = atomicAdd(job.block_done + blk, 1u) == (unsigned)(job.fx_chunks - 1) ? 1 : 0;
      __threadfence();
    }
    __syncthreads();
    if (*s_last == 0) return;
    if (threadIdx.x == 0) job.block_done[blk] = 0u;
#pragma unroll
    for (int k = 0; k < VD; ++k) sum[k].w[0] = sum[k].w[1] = sum[k].w[2] = sum[k].w[3] = 0u;
#pragma unroll 4
    for (int cc = 0; cc < job.fx_chunks; ++cc) {
#pragma unroll
      for (int k = 0; k < VD; ++k) {
        const uint4 a = __ldcg(p + ((size_t)cc * VD + k) * n_tgt + i);
        add128(sum[k].w, a.x, a.y, a.z, a.w);
      }
    }
  }
  if (i0 >= n_tgt) return;
  const int lx = job.fx[0].lx;  // one lambda per job
  double *o = job.out + (size_t)i0 * VD;
#pragma unroll
  for (int k = 0; k < VD; ++k) {
    u64 top = fx::pack64(sum[k].w[2], sum[k].w[3]), bot = fx::pack64(sum[k].w[0], sum[k].w[1]);
    const bool minus = (i64)top < 0;
    if (minus) {
      bot = 0ull - bot;
      top = ~top + (bot == 0ull ? 1ull : 0ull);
    }
    const double mag = fma((double)top, 18446744073709551616.0, (double)bot);
    const double val = minus ? -mag : mag;
    const double r = val * pow2(es - 91 - (k < 3 ? lx : 2 * lx)) * job.scale;
    o[k] = job.mode == OUT_ACCUMULATE ? o[k] + r : r;
  }
}

__device__ __forceinline__ bool takes(const QueueJob &job) {
  return job.fx_state != nullptr && job.fx_state->ok != 0;
}

// VDS: 9 for launches with segment targets among the jobs, 3 without.
template <int VDS, int FDA, int FDB, int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) rpy_fx_kernel(const QueueArgs q) {
  constexpr int kFx = 64 * Staged<(FDA > FDB ? FDA : FDB)>::words;
  constexpr int kF64 = 2 * kFp64Tile * Rec<double, (FDA > FDB ? FDA : FDB)>::len;
  __shared__ __align__(16) unsigned smem[kFx > kF64 ? kFx : kF64];
  __shared__ int s_end[kQueueMaxJobs];
  __shared__ int s_unit, s_last;
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int j = 0; j < q.n_jobs; ++j) {
      const QueueJob &jb = q.jobs[j];
      const bool skip = jb.skip != nullptr && *jb.skip != 0;
      acc += skip ? 0 : (jb.n_tgt + BLOCK - 1) / BLOCK * (takes(jb) ? jb.fx_chunks : jb.n_chunks);
      s_end[j] = acc;
    }
  }
  __syncthreads();
  const int n_units = q.n_jobs > 0 ? s_end[q.n_jobs - 1] : 0;
  for (;;) {
    if (threadIdx.x == 0) s_unit = (int)atomicAdd(q.counters, 1u);
    __syncthreads();
    const int u = s_unit;
    if (u >= n_units) break;
    int lo = 0, hi = q.n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_end[mid] > u) hi = mid; else lo = mid + 1;
    }
    const QueueJob &job = q.jobs[lo];
    const int local = u - (lo > 0 ? s_end[lo - 1] : 0);
    const bool fixed = takes(job);
    const int nc = fixed ? job.fx_chunks : job.n_chunks;
    const int blk = local / nc, c = local - blk * nc;
    if (VDS == 9 && job.vd == 6) {
      if (fixed)
        fx_unit<6, FDA, FDB, BLOCK>(job, blk, c, smem, &s_last);
      else
        queue_unit<double, 6, FDA, FDB, BLOCK, 1, kFp64Tile, false>(
            job, blk, c, reinterpret_cast<double *>(smem), nullptr, &s_last);
    } else {
      if (fixed)
        fx_unit<3, FDA, FDB, BLOCK>(job, blk, c, smem, &s_last);
      else
        queue_unit<double, 3, FDA, FDB, BLOCK, 1, kFp64Tile, false>(
            job, blk, c, reinterpret_cast<double *>(smem), nullptr, &s_last);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(q.counters + 1, 1u) == gridDim.x - 1) {
      q.counters[0] = 0u;
      q.counters[1] = 0u;
    }
  }
}

template <int VDS, int FDA, int FDB, int BLOCK, int MINB>
cudaError_t fx_launch(const QueueArgs &a, long long units, cudaStream_t st) {
  static std::atomic<int> occupancy[kMaxDevices];
  auto kern = rpy_fx_kernel<VDS, FDA, FDB, BLOCK, MINB>;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  int occ = occupancy[dev].load();
  if (occ == 0) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BLOCK, 0);
    if (e != cudaSuccess) return e;
    occupancy[dev].store(occ = occ < 1 ? 1 : occ);
  }
  const long long slots = (long long)occ * num_sms();
  kern<<<(int)(units < slots ? units : slots), BLOCK, 0, st>>>(a);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

int fx_lambda_exponent(double ai, double aj) { return ilogb(0.74 * (ai + aj)); }

static void fx_chunking(int n_a, int n_b, int n_particles, int *chunk, int *n_chunks) {
  const int tiles = (n_a + 31) / 32 + (n_b + 31) / 32;
  const long blocks = std::max(1L, ((long)n_particles + 127) / 128);
  const long want = std::max(1L, std::min<long>(kFxMaxChunks, (8192 + blocks - 1) / blocks));
  const int c = std::max(1, (int)((tiles + want - 1) / want));
  *chunk = c;
  *n_chunks = tiles > 0 ? (tiles + c - 1) / c : 0;
}

bool fx_job(QueueJob *j, FxState *state, const long long *tgt, const FxSource &a, const FxSource &b,
            int n_particles, int lx_min) {
  j->fx_state = nullptr;
  j->fx[0] = a;
  j->fx[1] = b;
  const double ra = j->a_a, rb = j->n_b > 0 ? j->a_b : j->a_a;
  // one lambda per job, of its smaller contact distance
  const int lx = fx_lambda_exponent(j->a_tgt, std::min(ra, rb));
  if (std::abs(lx) > kFxLambda || std::abs(lx_min) > kFxLambda) return false;
  for (int set = 0; set < 2; ++set) {
    const double at = ldexp(j->a_tgt, -lx), as = ldexp(set == 0 ? ra : rb, -lx);
    FxSource &f = j->fx[set];
    f.lx = lx;
    f.tshift = lx - lx_min;
    // widened by 2^-18: the FP32 r^2 it is compared with is within 2^-18.6 (at
    // contact in the widest frame, where the separation's words have 21 bits)
    f.near_q = (float)((at + as) * (at + as) * (1.0 + 3.8147e-6));
    const double sq = (at * at + as * as) / 3.0;
    if (!(sq < 3.9)) return false;  // radii too far apart for one lambda
    f.s = fx::limb_of((i64)rint(ldexp(sq, 61)));
  }
  j->fx_tgt = tgt;
  j->fx_state = state;
  fx_chunking(j->n_a, j->n_b, n_particles, &j->fx_chunk, &j->fx_chunks);
  return true;
}

cudaError_t launch_fx_pack(const FxSystem &q, cudaStream_t st) {
  const int tiles = (q.n[0] + 31) / 32 + (q.n[1] + 31) / 32;
  if (tiles == 0) return cudaSuccess;
  constexpr int per = kFxPackThreads / 32;
  fx_pack_kernel<<<(tiles + per - 1) / per, kFxPackThreads, 0, st>>>(q);
  count_launch();
  return cudaGetLastError();
}

// Threads per CTA by the variant: 0 picks by the units (below), 1 and 2 pin 64
// and 128. The launch's shape changes no bit of a result.
const QueueVariant g_qvariants_f64[kNumQueueVariantsF64] = {
    {0, 1, 64, 0}, {64, 1, 64, 8}, {128, 1, 64, 4}};

// Threads per CTA: 128 share a staged tile better, 64 split the work finer
// where there are fewer than eight units of 128 targets per SM: medium
// swimmer, M_ss (100 x 34 units) 3.68 ms with 128; M_bb of 1 289 blobs
// (11 x 41 units) 37 us with 64.
cudaError_t launch_fx(int variant, int sources, const QueueJob *jobs, const QueueJob *jobs_host,
                      int n_jobs, unsigned *counters, cudaStream_t st) {
  long long units[2] = {0, 0};
  bool has6 = false;
  for (int j = 0; j < n_jobs; ++j) {
    const QueueJob &q = jobs_host[j];
    // whichever form the device picks
    const int nc = q.fx_state == nullptr ? q.n_chunks : std::max(q.n_chunks, q.fx_chunks);
    for (int b = 0; b < 2; ++b) units[b] += (long long)((q.n_tgt + 64 * (b + 1) - 1) / (64 * (b + 1))) * nc;
    has6 = has6 || q.vd == 6;
  }
  if (units[0] <= 0) return cudaSuccess;
  const QueueArgs a{jobs, n_jobs, counters};
  const bool small = variant == 1 || (variant == 0 && units[1] < 8LL * num_sms());
  const long long u = units[small ? 0 : 1];
  if (sources == Q_SEG_BLOB)
    return small ? fx_launch<9, 6, 3, 64, 8>(a, u, st) : fx_launch<9, 6, 3, 128, 4>(a, u, st);
  if (sources == Q_SEG) {
    if (has6) return small ? fx_launch<9, 6, 0, 64, 8>(a, u, st) : fx_launch<9, 6, 0, 128, 4>(a, u, st);
    return small ? fx_launch<3, 6, 0, 64, 8>(a, u, st) : fx_launch<3, 6, 0, 128, 4>(a, u, st);
  }
  if (has6) return small ? fx_launch<9, 3, 0, 64, 8>(a, u, st) : fx_launch<9, 3, 0, 128, 4>(a, u, st);
  return small ? fx_launch<3, 3, 0, 64, 8>(a, u, st) : fx_launch<3, 3, 0, 128, 4>(a, u, st);
}

}  // namespace tfs
