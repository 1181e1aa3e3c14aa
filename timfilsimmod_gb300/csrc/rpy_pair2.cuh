// rpy_pair2.cuh -- FP32 pair sums on the packed FP32x2 instructions (FFMA2,
// FMUL2, FADD2), two sources per instruction.
//
// A packed instruction takes the FMA pipe the same two cycles as the two plain
// ones it replaces, but one issue slot instead of two, which leaves the slots
// that the compares, the reciprocal square roots and the shared-memory loads
// of a pair need: the plain form (58 instructions a 6x6 pair, 48 of them on
// the FMA pipe) was bound by issue at 0.58 of the FMA pipe's rate. Packing two
// sources of one target, not two targets of one source, keeps the shared
// loads at one copy of each source value (the target's position is the
// duplicated operand, held in registers): a 16-byte broadcast load occupies a
// sub-partition's share of the shared-memory port for 16 cycles, so
// duplicated source values bound the kernel by themselves.
//
// Sources are staged as pairs (2p, 2p + 1) with every component of the two side
// by side and the position negated: {-x -x' -y -y' | -z -z' F0 F0' | F1 F1' F2
// F2' | T0 T0' T1 T1' | T2 T2'}. An odd last source is paired with one at 1e15
// without force. The even and odd sources have sums of their own, added once
// per tile; the negative terms of the cross products too (a packed FMA cannot
// negate an operand), so no instruction is spent on signs.
//
// The far field with c1 = 1 - 3 s/r^2 and e = d/r^3 (47 packed operations for a
// 6x6 pair of two, against 48 for the form of tfs_device.cuh):
//   v_t += A F + c1 (d.F) e + T x e,  v_r += F x e - T/(2 r^3) + 3/(2 r^2) (d.T) e
// Pairs at or inside contact get 1/r = 0; the smallest r^2 of a tile says
// whether the lane rescans it for them.
//
// Measured, before (one source at a time) and after: grand mobility of the
// medium swimmer (12 800 segments, 2 562 blobs) 463 and 390 us, of the large one
// (80 000, 10 242) 14.3 and 11.8 ms -- 56 cycles a 6x6 pair, warp and
// sub-partition, of which the FMA pipe takes 47 --, the 3x3 products of 15 362
// particles 254 and 204 us; the error against 64-bit sums falls from 9.1e-7 to
// 8.1e-7 (large) as each half of the sources has a sum of its own. Two targets
// a thread, a clamp of r^2 in place of the compare and select, separate sums
// for the terms with factors 1/2 and 3/2, and unrolling by two were each within
// 3% of this form.
#pragma once

#include <cuda_runtime.h>

#include "rpy_tile.cuh"

namespace tfs {

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }

template <int FD>
struct Pair2 {
  static constexpr int len = FD == 6 ? 20 : 12;  // floats of two sources
};

// Sums of one target: positive and negative terms, even and odd sources.
template <int VD, int FD>
struct Sum2 {
  static constexpr bool kTorque = FD == 6, kRot = VD == 6;
  float2 t[3], tn[kTorque ? 3 : 1], r[kRot ? 3 : 1], rn[kRot ? 3 : 1];
  __device__ __forceinline__ void zero() {
    const float2 z = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      t[k] = z;
      if (kTorque) tn[kTorque ? k : 0] = z;
      if (kRot) r[kRot ? k : 0] = rn[kRot ? k : 0] = z;
    }
  }
  __device__ __forceinline__ float get(int k) const {
    if (k < 3) {
      const float s = t[k].x + t[k].y;
      if constexpr (kTorque) return s - (tn[k].x + tn[k].y);
      return s;
    }
    if constexpr (kRot) return (r[k - 3].x + r[k - 3].y) - (rn[k - 3].x + rn[k - 3].y);
    return 0.f;
  }
};

template <int VD, int FD>
__device__ __forceinline__ void far_pair2(Sum2<VD, FD> &v, float2 dx, float2 dy, float2 dz,
                                          float2 rm1, const float2 (&f)[FD], float2 s, float2 s3) {
  const float2 rm2 = mul2(rm1, rm1);
  const float2 rm3 = mul2(rm1, rm2);
  const float2 A = fma2(s, rm3, rm1);
  const float2 c1 = fma2(s3, rm2, both(1.f));
  const float2 dF = fma2(dx, f[0], fma2(dy, f[1], mul2(dz, f[2])));
  float2 c = mul2(c1, dF);
  if constexpr (VD == 3 && FD == 3) {
    c = mul2(c, rm3);
    v.t[0] = fma2(A, f[0], fma2(c, dx, v.t[0]));
    v.t[1] = fma2(A, f[1], fma2(c, dy, v.t[1]));
    v.t[2] = fma2(A, f[2], fma2(c, dz, v.t[2]));
  } else {
    const float2 ex = mul2(rm3, dx), ey = mul2(rm3, dy), ez = mul2(rm3, dz);
    v.t[0] = fma2(A, f[0], fma2(c, ex, v.t[0]));
    v.t[1] = fma2(A, f[1], fma2(c, ey, v.t[1]));
    v.t[2] = fma2(A, f[2], fma2(c, ez, v.t[2]));
    if constexpr (FD == 6) {
      v.t[0] = fma2(f[4], ez, v.t[0]);
      v.tn[0] = fma2(f[5], ey, v.tn[0]);
      v.t[1] = fma2(f[5], ex, v.t[1]);
      v.tn[1] = fma2(f[3], ez, v.tn[1]);
      v.t[2] = fma2(f[3], ey, v.t[2]);
      v.tn[2] = fma2(f[4], ex, v.tn[2]);
    }
    if constexpr (VD == 6) {
      v.r[0] = fma2(f[1], ez, v.r[0]);
      v.rn[0] = fma2(f[2], ey, v.rn[0]);
      v.r[1] = fma2(f[2], ex, v.r[1]);
      v.rn[1] = fma2(f[0], ez, v.rn[1]);
      v.r[2] = fma2(f[0], ey, v.r[2]);
      v.rn[2] = fma2(f[1], ex, v.rn[2]);
      if constexpr (FD == 6) {
        const float2 h = mul2(both(0.5f), rm3);
        const float2 dT = fma2(dx, f[3], fma2(dy, f[4], mul2(dz, f[5])));
        const float2 q = mul2(mul2(both(1.5f), rm2), dT);
        v.r[0] = fma2(q, ex, v.r[0]);
        v.rn[0] = fma2(h, f[3], v.rn[0]);
        v.r[1] = fma2(q, ey, v.r[1]);
        v.rn[1] = fma2(h, f[4], v.rn[1]);
        v.r[2] = fma2(q, ez, v.r[2]);
        v.rn[2] = fma2(h, f[5], v.rn[2]);
      }
    }
  }
}

// Stage the records [base, base + cnt) as interleaved pairs; no barrier.
template <int FD, int BLOCK>
__device__ __forceinline__ void stage_pairs(const float *__restrict__ rec, int base, int cnt,
                                            float *smem) {
  constexpr int L = Rec<float, FD>::len, W = Pair2<FD>::len;
  for (int j = threadIdx.x; j < cnt; j += BLOCK) {
    const float4 *q = reinterpret_cast<const float4 *>(rec + (size_t)(base + j) * L);
    float *o = smem + (j >> 1) * W + (j & 1);
    const float4 a = __ldg(q), b = __ldg(q + 1);
    o[0] = -a.x;
    o[2] = -a.y;
    o[4] = -a.z;
    o[6] = a.w;
    o[8] = b.x;
    o[10] = b.y;
    if (FD == 6) {
      o[12] = b.z;
      o[14] = b.w;
      o[16] = __ldg(rec + (size_t)(base + j) * L + 8);
    }
  }
  if ((cnt & 1) && threadIdx.x < FD + 3)  // the odd last source's partner
    smem[(cnt >> 1) * W + 1 + 2 * threadIdx.x] = threadIdx.x < 3 ? 1e15f : 0.f;
}

// One pair of staged sources: negated positions, forces (and torques).
template <int FD>
__device__ __forceinline__ void load_pair(const float *o, float2 &nx, float2 &ny, float2 &nz,
                                          float2 (&f)[FD]) {
  const float4 *q = reinterpret_cast<const float4 *>(o);
  const float4 a = q[0], b = q[1], c = q[2];
  nx = make_float2(a.x, a.y);
  ny = make_float2(a.z, a.w);
  nz = make_float2(b.x, b.y);
  f[0] = make_float2(b.z, b.w);
  f[1] = make_float2(c.x, c.y);
  f[2] = make_float2(c.z, c.w);
  if constexpr (FD == 6) {
    const float4 d = q[3];
    f[3] = make_float2(d.x, d.y);
    f[4] = make_float2(d.z, d.w);
    f[5] = *reinterpret_cast<const float2 *>(q + 4);
  }
}

// The sources [lo, hi) of one FP32 record array into the compensated sums of
// this thread's targets (hl, as Comp<float>). compute = false (warp-uniform):
// the warp has no target of its own and only helps stage the tiles.
template <int VD, int FD, int BLOCK, int TPT, int TS>
__device__ __forceinline__ void sum_source_range2(const float (&xt)[TPT], const float (&yt)[TPT],
                                                  const float (&zt)[TPT],
                                                  const float *__restrict__ rec, int lo, int hi,
                                                  const PairConst<float> &pc, float *smem, float *hl,
                                                  bool compute) {
  constexpr int W = Pair2<FD>::len;
  const float2 s = both(pc.s), s3 = both(pc.s3);
  for (int base = lo; base < hi; base += TS) {
    const int cnt = min(TS, hi - base);
    __syncthreads();  // previous tile fully consumed
    stage_pairs<FD, BLOCK>(rec, base, cnt, smem);
    __syncthreads();
    if (!compute) continue;
    Sum2<VD, FD> v[TPT];
    float rmin[TPT];
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
      v[t].zero();
      rmin[t] = INFINITY;
    }
    const int pairs = (cnt + 1) >> 1;
#pragma unroll 1
    for (int p = 0; p < pairs; ++p) {
      float2 nx, ny, nz, f[FD];
      load_pair<FD>(smem + p * W, nx, ny, nz, f);
#pragma unroll
      for (int t = 0; t < TPT; ++t) {
        const float2 dx = add2(both(xt[t]), nx);
        const float2 dy = add2(both(yt[t]), ny);
        const float2 dz = add2(both(zt[t]), nz);
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        rmin[t] = fminf(rmin[t], fminf(r2.x, r2.y));
        float2 rm1;
        rm1.x = r2.x > pc.asum2 ? rsqrt_far(r2.x) : 0.f;
        rm1.y = r2.y > pc.asum2 ? rsqrt_far(r2.y) : 0.f;
        far_pair2<VD, FD>(v[t], dx, dy, dz, rm1, f, s, s3);
      }
    }
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
      float n[VD];
#pragma unroll
      for (int k = 0; k < VD; ++k) n[k] = 0.f;
      // (a NaN separation compares false both times, as in the far pass)
      if (!(rmin[t] > pc.asum2)) {
        for (int j = 0; j < cnt; ++j) {
          const float *o = smem + (j >> 1) * W + (j & 1);
          float g[FD];
          const float dx = xt[t] + o[0], dy = yt[t] + o[2], dz = zt[t] + o[4];
          const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
          if (r2 > pc.asum2) continue;
#pragma unroll
          for (int k = 0; k < FD; ++k) g[k] = o[6 + 2 * k];
          near_pair<float, VD, FD>(n, dx, dy, dz, r2, g, pc);
        }
      }
#pragma unroll
      for (int k = 0; k < VD; ++k) {
        float *hp = hl + ((t * VD + k) * 2) * BLOCK + threadIdx.x, *lp = hp + BLOCK;
        float h = *hp, l = *lp;
        two_sum(h, l, v[t].get(k));
        two_sum(h, l, n[k]);
        *hp = h;
        *lp = l;
      }
    }
  }
}

}  // namespace tfs
