// rpy_bb64.cu -- the FP64 blob-blob product of the kernel-sequence GMRES.
//
// The same sums as rpy_tile_kernel<double, 3, 3>, bit for bit: source splits
// of the same size, tiles of 128 sources, every far pair added in source
// order and the pairs of a tile inside the contact distance after it, again
// in source order. A warm-started FP64 GMRES amplifies a difference of 1e-14
// in its product up to 1e5 times, so the order of the sums is part of the
// result.
//
// What bounds it: FP64 instructions, 64 to 78 cycles each on an SM
// sub-partition whatever the number of active lanes. The tile kernel keeps a
// target's whole sum on one thread, so its source splits (a tile at least)
// leave it 36 CTAs at 642 blobs. Only the additions are serial, though: the
// 21 instructions of a pair's scalars A, B (d.F) and d (far_pair) are not.
// Here a CTA's warps compute those for 32 sources (a lane each) of one target
// after another into shared memory, and up to three warps, one lane per
// (target, component), run the ordered sums of the stage before. Their two
// instructions a source serve 32 chains at once, so the split costs nothing:
// 642 blobs 184 -> 33.6 us, 1 289 blobs 177 -> 103 us.
#include <atomic>

#include <algorithm>

#include "rpy_tile.cuh"

namespace tfs {

constexpr int kBbBlock = 256;
constexpr int kBbStage = 32;             // sources per stage: one per lane
constexpr int kBbTile = 128;             // sources between two near passes
constexpr int kBbMaxTargets = 32;        // per CTA
constexpr int kBbRow = kBbStage + 1;     // doubles; odd, so lanes of different targets
                                         // read different banks

// Doubles of one stage buffer for nt targets: A, B (d.F), dx, dy, dz of every
// pair, then the forces of the sources.
__host__ __device__ constexpr int bb_stage_elems(int nt) {
  return 5 * nt * kBbRow + 3 * kBbStage;
}

__global__ void __launch_bounds__(kBbBlock, 2) rpy_bb64_kernel(const TileArgs args, int nt,
                                                              double a_self) {
  extern __shared__ __align__(16) double bb_smem[];
  __shared__ double xt[3][kBbMaxTargets];
  __shared__ unsigned near[2][kBbMaxTargets][kBbTile / kBbStage];
  __shared__ int next[2];
  if (args.skip != nullptr && *args.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = blockIdx.x * nt, cnt = min(nt, args.n_tgt - t0);
  const int s0 = blockIdx.y * args.chunk, s1 = min(s0 + args.chunk, args.n_a);
  const int stages = (s1 - s0 + kBbStage - 1) / kBbStage;
  const double *rec = reinterpret_cast<const double *>(args.src_a);
  PairConst<double> pc;
  pc.ai = args.a_tgt;
  pc.aj = args.a_a;
  pc.asum2 = (args.a_tgt + args.a_a) * (args.a_tgt + args.a_a);
  pc.s = (args.a_tgt * args.a_tgt + args.a_a * args.a_a) / 3.0;
  pc.s3 = -(args.a_tgt * args.a_tgt + args.a_a * args.a_a);
  for (int q = tid; q < 3 * cnt; q += kBbBlock) xt[q % 3][q / 3] = args.x_tgt[3 * (size_t)t0 + q];
  if (tid < 2) next[tid] = 0;

  const int row = nt * kBbRow;
  const int q = tid, qt = q / 3, qc = q - 3 * qt;  // this lane's chain: target, component
  const bool chain = q < 3 * cnt;
  const bool chain_warp = 32 * warp < 3 * cnt;
  double v = 0.0;

  for (int s = 0; s <= stages; ++s) {
    __syncthreads();  // stage s-1 is produced, stage s-2's buffer is free
    if (tid == 0) next[(s + 1) & 1] = 0;
    if (s > 0 && chain_warp) {
      const double *buf = bb_smem + ((s - 1) & 1) * bb_stage_elems(nt);
      const int base = s0 + (s - 1) * kBbStage, n = min(kBbStage, s1 - base);
      if (chain) {
        const double *A = buf + qt * kBbRow, *B = A + row, *d = B + (1 + qc) * row;
        const double *f = buf + 5 * row + qc;
#pragma unroll 4
        for (int j = 0; j < n; ++j) v = fma(A[j], f[3 * j], fma(B[j], d[j], v));
        if (s == stages || s % (kBbTile / kBbStage) == 0) {
          const int tile = (s - 1) / (kBbTile / kBbStage);
          for (int w = 0; w <= (s - 1) % (kBbTile / kBbStage); ++w) {
            for (unsigned m = near[tile & 1][qt][w]; m != 0u; m &= m - 1u) {
              const int j = s0 + tile * kBbTile + w * kBbStage + __ffs(m) - 1;
              double sx, sy, sz, f3[3];
              RecLoad<double, 3>::get(rec + (size_t)j * 6, sx, sy, sz, f3);
              const double dx = xt[0][qt] - sx, dy = xt[1][qt] - sy, dz = xt[2][qt] - sz;
              const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
              if (r2 == 0.0) {  // near_pair at r = 0: (A f + 0)
                v = v + __dmul_rn(a_self, qc == 0 ? f3[0] : qc == 1 ? f3[1] : f3[2]);
              } else {
                double u[3] = {0.0, 0.0, 0.0};
                near_pair<double, 3, 3>(u, dx, dy, dz, r2, f3, pc);
                v = v + (qc == 0 ? u[0] : qc == 1 ? u[1] : u[2]);
              }
            }
          }
        }
      }
    }
    if (s == stages) break;
    double *buf = bb_smem + (s & 1) * bb_stage_elems(nt);
    const int j = s0 + s * kBbStage + lane;
    double sx = 0.0, sy = 0.0, sz = 0.0, f[3] = {0.0, 0.0, 0.0};
    if (j < s1) RecLoad<double, 3>::get(rec + (size_t)j * 6, sx, sy, sz, f);
    if (warp == kBbBlock / 32 - 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) buf[5 * row + 3 * lane + k] = f[k];
    }
    for (;;) {
      int t = lane == 0 ? atomicAdd(&next[s & 1], 1) : 0;
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t >= cnt) break;
      const double dx = xt[0][t] - sx, dy = xt[1][t] - sy, dz = xt[2][t] - sz;
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      const bool far = r2 > pc.asum2;
      const double rs = rsqrt_far(r2);
      const double rm1 = far ? rs : 0.0;
      const double rm2 = rm1 * rm1;
      const double rm3 = rm1 * rm2;
      const double rm5 = rm3 * rm2;
      const double dF = fma(dx, f[0], fma(dy, f[1], dz * f[2]));
      double *o = buf + t * kBbRow + lane;
      o[0] = fma(pc.s, rm3, rm1);
      o[row] = fma(pc.s3, rm5, rm3) * dF;
      o[2 * row] = dx;
      o[3 * row] = dy;
      o[4 * row] = dz;
      const unsigned m = __ballot_sync(0xffffffffu, !far && j < s1);
      if (lane == 0) near[(s / (kBbTile / kBbStage)) & 1][t][s % (kBbTile / kBbStage)] = m;
    }
  }
  if (!chain) return;
  const double r = args.scale * v;
  double *o = args.out + (args.mode == OUT_PARTIAL ? 3 * (size_t)blockIdx.y * args.n_tgt : 0) +
              3 * (size_t)t0 + q;
  if (args.mode == OUT_ACCUMULATE) *o += r;
  else *o = r;
}

// Targets per CTA: the fewest FP64 instructions on the busiest SM. A CTA
// issues, per 128 sources, 21 a target and 4 stages for the pair scalars and
// 256 a chain warp for the sums; its 3 chains a target fill warps of 32 best
// at 10, 21 or 32 targets, the SMs at a count that divides the targets well.
static int bb_targets(int n_tgt, int n_src, int chunk, int sms) {
  long best = 0;
  int nt_best = 1;
  for (int nt = 1; nt <= kBbMaxTargets; ++nt) {
    const long groups = (n_tgt + nt - 1) / nt;
    const long full = groups * (n_src / chunk), rest = groups * (n_src % chunk);
    const long ctas = full + (rest + chunk - 1) / chunk;
    const long cost = ((ctas + sms - 1) / sms) * (4 * 21 * nt + 256 * ((3 * nt + 31) / 32));
    if (best == 0 || cost <= best) {
      best = cost;
      nt_best = nt;
    }
  }
  return nt_best;
}

cudaError_t launch_bb64(const TileArgs &a, int splits, cudaStream_t st) {
  static std::atomic<int> ready[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  if (ready[dev].load() == 0) {
    e = cudaFuncSetAttribute(rpy_bb64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * 8 * bb_stage_elems(kBbMaxTargets));
    if (e != cudaSuccess) return e;
    ready[dev].store(1);
  }
  const int nt = bb_targets(a.n_tgt, a.n_a, a.chunk, num_sms());
  const dim3 grid((a.n_tgt + nt - 1) / nt, splits);
  rpy_bb64_kernel<<<grid, kBbBlock, 2 * 8 * bb_stage_elems(nt), st>>>(
      a, nt, 4.0 / (3.0 * std::max(a.a_tgt, a.a_a)));
  return cudaGetLastError();
}

}  // namespace tfs
