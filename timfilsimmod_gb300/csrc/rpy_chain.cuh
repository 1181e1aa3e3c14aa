// rpy_chain.cuh -- FP64 pair sums of a source chunk for a few targets, bit for
// bit those of sum_source_range (rpy_tile.cuh: 128-source tiles, every far
// pair in source order, then the tile's pairs inside the contact distance),
// with the work of one target spread over a CTA.
//
// What bounds them: FP64 instructions, 64 to 78 cycles each on an SM
// sub-partition whatever the number of active lanes. The tile form keeps a
// target's whole sum on one thread, so a product of few targets leaves most
// SMs idle: source chunks can't be cut finer without changing the sums. Only
// the additions are serial, though; a pair's scalars -- A, B (d.F), d and, with
// torques, d/r^3 and the torque factors (far_pair) -- are not. A CTA's warps
// compute those for 32 sources (a lane each) of one target after another into
// shared memory, and up to three warps, one lane per (target, component), run
// the ordered sums of the stage before. Their instructions serve 32 sums at
// once, so the split costs nothing. The scalars' plain products run on the
// integer pipe beside (soft_mul.cuh), which leaves 12 FP64 instructions of 21
// for the scalars of a 3x3 pair, 14 of 29 of a 6x6 pair.
#pragma once

#include "rpy_tile.cuh"
#include "soft_mul.cuh"

namespace tfs {

constexpr int kChainBlock = 256;               // (192, 320, 384: 6, 3 and 9% slower)
constexpr int kChainStage = 32;               // sources per stage: one per lane
constexpr int kChainTile = 128;               // sources between two near passes
constexpr int kChainStages = kChainTile / kChainStage;
constexpr int kChainMaxTargets = 32;
constexpr int kChainRow = kChainStage + 1;    // doubles; odd, so lanes of different
                                              // targets read different banks

// Pair scalars kept per (target, source): A, B (d.F), d; d/r^3; the torque's.
template <int VD, int FD>
struct ChainFields {
  static constexpr int n = VD == 6 && FD == 6 ? 10 : VD == 6 || FD == 6 ? 8 : 5;
  // FP64 instructions of a pair's scalars (beside the integer products), and of a
  // sum's step
  static constexpr int scalars = 12 + (VD == 6 && FD == 6 ? 2 : 0);
  static constexpr int steps = VD == 6 && FD == 6 ? 4 : FD == 6 ? 4 : 2;
  static constexpr int forces = VD == 3 && FD == 3 ? 3 : 2 * FD;  // rows: F, T and, negated, again
};

// Doubles of one stage buffer for nt targets: the fields of every pair, then
// the forces of the sources.
template <int VD, int FD>
__host__ __device__ constexpr int chain_stage_elems(int nt) {
  return (ChainFields<VD, FD>::n * nt + ChainFields<VD, FD>::forces) * kChainRow;
}

struct ChainShared {
  double xt[3][kChainMaxTargets];
  unsigned near[2][kChainMaxTargets][kChainStages];  // by tile parity: sources inside contact
  int next[2];
};

// far_pair's scalars of target t and this lane's source into o (row doubles
// from field to field). SOFT: the products on the integer pipe (soft_mul.cuh),
// which runs beside the FP64 pipe -- 8 of the 20 FP64 instructions of a 3x3
// pair's scalars and the compare, 15 of 28 of a 6x6 pair's; !ok: one of them is
// out of its range, and the scalars are to be computed without.
template <int VD, int FD, bool SOFT>
__device__ __forceinline__ void pair_scalars(const ChainShared &sh, int t, double sx, double sy,
                                             double sz, const double (&f)[FD],
                                             const PairConst<double> &pc, double *o, int row,
                                             bool &far, bool &ok) {
  auto mul = [&](double a, double b) { return SOFT ? soft::mul(a, b, &ok) : a * b; };
  const double dx = sh.xt[0][t] - sx, dy = sh.xt[1][t] - sy, dz = sh.xt[2][t] - sz;
  const double r2 = fma(dx, dx, fma(dy, dy, mul(dz, dz)));
  if constexpr (SOFT) {
    // numbers not below zero compare as their bits do; a NaN is above infinity
    const long long u = __double_as_longlong(r2);
    far = u > __double_as_longlong(pc.asum2) && u <= 0x7ff0000000000000ll;
  } else {
    far = r2 > pc.asum2;
  }
  const double rs = rsqrt_far(r2, mul);
  const double rm1 = far ? rs : 0.0;
  const double rm2 = mul(rm1, rm1);
  const double rm3 = mul(rm1, rm2);
  const double rm5 = mul(rm3, rm2);
  const double dF = fma(dx, f[0], fma(dy, f[1], mul(dz, f[2])));
  o[0] = fma(pc.s, rm3, rm1);
  o[row] = mul(fma(pc.s3, rm5, rm3), dF);
  o[2 * row] = dx;
  o[3 * row] = dy;
  o[4 * row] = dz;
  if constexpr (VD == 6 || FD == 6) {
    o[5 * row] = mul(rm3, dx);
    o[6 * row] = mul(rm3, dy);
    o[7 * row] = mul(rm3, dz);
  }
  if constexpr (VD == 6 && FD == 6) {
    const double dT = fma(dx, f[3], fma(dy, f[4], mul(dz, f[5])));
    o[8 * row] = mul(-0.5, rm3);
    o[9 * row] = mul(mul(1.5, rm5), dT);
  }
}

// The sum of the lane's (target, component) -- target threadIdx.x / VD, component
// threadIdx.x % VD, for threadIdx.x < VD cnt -- over the sources [s0, s1) of rec.
// sh.xt holds the targets' positions (a barrier follows in here); a_self,
// a_self_rot: the self term's coefficients 4/(3 a), 1/a^3. buf: two stage
// buffers. Ends without a barrier.
template <int VD, int FD>
__device__ __forceinline__ double chain_sums(ChainShared &sh, const double *__restrict__ rec,
                                             int s0, int s1, int cnt, int nt,
                                             const PairConst<double> &pc, double a_self,
                                             double a_self_rot, double *buf2) {
  using Fld = ChainFields<VD, FD>;
  constexpr int L = Rec<double, FD>::len;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int stages = (s1 - s0 + kChainStage - 1) / kChainStage;
  const int row = nt * kChainRow;
  const int qt = tid / VD, qc = tid - VD * qt;
  const bool chain = tid < VD * cnt, chain_warp = 32 * warp < VD * cnt;
  const int k = qc % 3, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
  // offsets of the factors of this lane's steps in a stage buffer
  int xo[Fld::steps], yo[Fld::steps];
  {
    const int fo = Fld::n * row;  // force rows
    auto field = [&](int f) { return f * row + qt * kChainRow; };
    auto force = [&](int r) { return fo + r * kChainRow; };
    if (qc < 3) {
      xo[0] = field(1);
      yo[0] = field(2 + k);
      xo[1] = field(0);
      yo[1] = force(k);
      if constexpr (FD == 6) {
        xo[2] = field(5 + k1);
        yo[2] = force(6 + 3 + k2);  // negated
        xo[3] = field(5 + k2);
        yo[3] = force(3 + k1);
      }
    } else if constexpr (VD == 6) {
      xo[0] = field(5 + k1);
      yo[0] = force(FD + k2);
      xo[1] = field(5 + k2);
      yo[1] = force(k1);
      if constexpr (FD == 6) {
        xo[2] = field(9);
        yo[2] = field(2 + k);
        xo[3] = field(8);
        yo[3] = force(3 + k);
      }
    }
  }
  if (tid < 2) sh.next[tid] = 0;
  double v = 0.0;
  for (int s = 0; s <= stages; ++s) {
    __syncthreads();  // stage s-1 is produced, stage s-2's buffer is free
    if (tid == 0) sh.next[(s + 1) & 1] = 0;
    if (s > 0 && chain_warp && chain) {
      const double *buf = buf2 + ((s - 1) & 1) * chain_stage_elems<VD, FD>(nt);
      const int n = min(kChainStage, s1 - s0 - (s - 1) * kChainStage);
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
#pragma unroll
        for (int u = 0; u < Fld::steps; ++u) v = fma(buf[xo[u] + j], buf[yo[u] + j], v);
      }
      if (s == stages || s % kChainStages == 0) {
        const int tile = (s - 1) / kChainStages;
        for (int w = 0; w <= (s - 1) % kChainStages; ++w) {
          for (unsigned m = sh.near[tile & 1][qt][w]; m != 0u; m &= m - 1u) {
            const int j = s0 + tile * kChainTile + w * kChainStage + __ffs(m) - 1;
            double sx, sy, sz, f[FD];
            RecLoad<double, FD>::get(rec + (size_t)j * L, sx, sy, sz, f);
            const double dx = sh.xt[0][qt] - sx, dy = sh.xt[1][qt] - sy, dz = sh.xt[2][qt] - sz;
            const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
            if (r2 == 0.0) {
              // near_pair at r = 0: 4/(3a) F and 1/a^3 T, its other terms zero
              if (qc < 3) v = v + __dmul_rn(a_self, k == 0 ? f[0] : k == 1 ? f[1] : f[2]);
              else if constexpr (FD == 6)
                v = v + __dmul_rn(a_self_rot, k == 0 ? f[3] : k == 1 ? f[4] : f[5]);
            } else {
              double u[VD];
#pragma unroll
              for (int c = 0; c < VD; ++c) u[c] = c == qc ? v : 0.0;
              near_pair<double, VD, FD>(u, dx, dy, dz, r2, f, pc);
#pragma unroll
              for (int c = 0; c < VD; ++c) v = c == qc ? u[c] : v;
            }
          }
        }
      }
    }
    if (s == stages) break;
    double *buf = buf2 + (s & 1) * chain_stage_elems<VD, FD>(nt);
    const int j = s0 + s * kChainStage + lane;
    double sx = 0.0, sy = 0.0, sz = 0.0, f[FD] = {};
    if (j < s1) RecLoad<double, FD>::get(rec + (size_t)j * L, sx, sy, sz, f);
    if (warp == kChainBlock / 32 - 1) {
      double *o = buf + Fld::n * row + lane;
#pragma unroll
      for (int c = 0; c < FD; ++c) {
        o[c * kChainRow] = f[c];
        if (Fld::forces > FD) o[(FD + c) * kChainRow] = -f[c];
      }
    }
    for (;;) {
      int t = lane == 0 ? atomicAdd(&sh.next[s & 1], 1) : 0;
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t >= cnt) break;
      double *o = buf + t * kChainRow + lane;
      bool far, ok = true;
      pair_scalars<VD, FD, true>(sh, t, sx, sy, sz, f, pc, o, row, far, ok);
      // (a near pair has zero scalars, which the integer products take too)
      if (__any_sync(0xffffffffu, !ok && j < s1))
        pair_scalars<VD, FD, false>(sh, t, sx, sy, sz, f, pc, o, row, far, ok);
      const unsigned m = __ballot_sync(0xffffffffu, !far && j < s1);
      if (lane == 0) sh.near[(s / kChainStages) & 1][t][s % kChainStages] = m;
    }
  }
  return v;
}

}  // namespace tfs
