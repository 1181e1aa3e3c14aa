// rpy_bb64.cu -- FP64 products whose sums must keep the bits of the tile form
// (rpy_chain.cuh): the blob-blob product of the kernel-sequence
// GMRES and the plain work-queue jobs. A warm-started FP64 GMRES amplifies a
// difference of 1e-14 in its product up to 1e5 times, so the order of the sums
// is part of the result.
#include <atomic>

#include <algorithm>

#include "rpy_chain.cuh"

namespace tfs {

// rpy_tile_kernel<double, 3, 3, 0, ...> of 128-source tiles. 642 blobs 184 -> 28 us,
// 1 289 blobs 177 -> 73 us (34 and 103 us without the integer products).
__global__ void __launch_bounds__(kChainBlock, 2) rpy_bb64_kernel(const TileArgs args, int nt,
                                                                 double a_self) {
  extern __shared__ __align__(16) double bb_smem[];
  __shared__ ChainShared sh;
  if (args.skip != nullptr && *args.skip) return;
  const int tid = threadIdx.x;
  const int t0 = blockIdx.x * nt, cnt = min(nt, args.n_tgt - t0);
  const int s0 = blockIdx.y * args.chunk, s1 = min(s0 + args.chunk, args.n_a);
  PairConst<double> pc;
  pc.ai = args.a_tgt;
  pc.aj = args.a_a;
  pc.asum2 = (args.a_tgt + args.a_a) * (args.a_tgt + args.a_a);
  pc.s = (args.a_tgt * args.a_tgt + args.a_a * args.a_a) / 3.0;
  pc.s3 = -(args.a_tgt * args.a_tgt + args.a_a * args.a_a);
  for (int q = tid; q < 3 * cnt; q += kChainBlock)
    sh.xt[q % 3][q / 3] = args.x_tgt[3 * (size_t)t0 + q];
  const double v = chain_sums<3, 3>(sh, reinterpret_cast<const double *>(args.src_a), s0, s1, cnt,
                                    nt, pc, a_self, 0.0, bb_smem);
  if (tid >= 3 * cnt) return;
  const double r = args.scale * v;
  double *o = args.out + (args.mode == OUT_PARTIAL ? 3 * (size_t)blockIdx.y * args.n_tgt : 0) +
              3 * (size_t)t0 + tid;
  if (args.mode == OUT_ACCUMULATE) *o += r;
  else *o = r;
}

// Targets per CTA: the fewest FP64 instructions on the busiest SM. A CTA
// issues, per 128 sources, 12 a target and 4 stages for the pair scalars and
// 256 a chain warp for the sums; its 3 chains a target fill warps of 32 best
// at 10, 21 or 32 targets, the SMs at a count that divides the targets well.
static int bb_targets(int n_tgt, int n_src, int chunk, int sms) {
  using Fld = ChainFields<3, 3>;
  long best = 0;
  int nt_best = 1;
  for (int nt = 1; nt <= kChainMaxTargets; ++nt) {
    const long groups = (n_tgt + nt - 1) / nt;
    const long full = groups * (n_src / chunk), rest = groups * (n_src % chunk);
    const long ctas = full + (rest + chunk - 1) / chunk;
    const long cost = ((ctas + sms - 1) / sms) *
                      (kChainStages * Fld::scalars * nt +
                       kChainTile * Fld::steps * ((3 * nt + 31) / 32));
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
                             2 * 8 * chain_stage_elems<3, 3>(kChainMaxTargets));
    if (e != cudaSuccess) return e;
    ready[dev].store(1);
  }
  const int nt = bb_targets(a.n_tgt, a.n_a, a.chunk, num_sms());
  const dim3 grid((a.n_tgt + nt - 1) / nt, splits);
  rpy_bb64_kernel<<<grid, kChainBlock, 2 * 8 * chain_stage_elems<3, 3>(nt), st>>>(
      a, nt, 4.0 / (3.0 * std::max(a.a_tgt, a.a_a)));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Plain FP64 work-queue jobs (rpy_queue.cuh's queue_unit<double, ...>): units of
// kPlainTargets targets against one chunk, handed out by a counter; the
// chunk sums go to the job's partials, and the last unit of 32 targets (the
// granularity of the job's arrival counters) adds them in chunk order.
//
// Every plain FP64 launch takes this form, as it is the faster one at every
// size: M_ss with M_bs of 640 segments and 642 blobs 629 -> 101 us, M_sb 318 -> 52
// us, M_bs of 1 289 blobs on 3 587 segments 482 -> 309 us, on 6 000 634 -> 529,
// of 2 562 on 3 587 799 -> 605.
// ---------------------------------------------------------------------------
constexpr int kPlainTargets = 16;  // 96 sums of a segment target: three full warps

template <int VD, int FD>
__device__ __forceinline__ void plain_unit(const QueueJob &job, int grp, int c, ChainShared &sh,
                                           double *smem, int *s_last) {
  constexpr int L = Rec<double, VD == 6 ? 6 : 3>::len;
  const int tid = threadIdx.x, n_tgt = job.n_tgt;
  const int t0 = grp * kPlainTargets, cnt = min(kPlainTargets, n_tgt - t0);
  const int s0 = c * job.chunk, s1 = min(s0 + job.chunk, job.n_a);
  const double *q = job.pc64[0];
  PairConst<double> pc;
  pc.ai = q[0]; pc.aj = q[1]; pc.asum2 = q[2]; pc.s = q[3]; pc.s3 = q[4];
  const double *tgt = reinterpret_cast<const double *>(job.tgt_rec);
  for (int i = tid; i < 3 * cnt; i += kChainBlock)
    sh.xt[i % 3][i / 3] = tgt[(size_t)(t0 + i / 3) * L + i % 3];
  const double amax = fmax(pc.ai, pc.aj);
  const double v = chain_sums<VD, FD>(sh, reinterpret_cast<const double *>(job.src_a), s0, s1, cnt,
                                      kPlainTargets, pc, 4.0 / (3.0 * amax),
                                      1.0 / (amax * amax * amax), smem);
  const double sc = job.scale;
  if (job.n_chunks == 1) {
    if (tid < VD * cnt) {
      double *o = job.out + (size_t)t0 * VD + tid;
      const double r = sc * v;
      *o = job.mode == OUT_ACCUMULATE ? *o + r : r;
    }
    return;
  }
  double *part = reinterpret_cast<double *>(job.partial);
  const size_t stride = (size_t)n_tgt * VD;
  if (tid < VD * cnt) part[c * stride + (size_t)t0 * VD + tid] = v;
  const int blk = t0 / 32, b0 = 32 * blk, nb = min(32, n_tgt - b0);
  const unsigned arrivals = (unsigned)(job.n_chunks * ((nb + kPlainTargets - 1) / kPlainTargets));
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    *s_last = atomicAdd(job.block_done + blk, 1u) == arrivals - 1u ? 1 : 0;
    __threadfence();
  }
  __syncthreads();
  if (*s_last == 0) return;
  static_assert(kChainBlock >= 6 * 32, "a thread per component of 32 targets");
  if (tid < VD * nb) {
    const double *p = part + (size_t)b0 * VD + tid;
    double r = 0.0;
#pragma unroll 4
    for (int cc = 0; cc < job.n_chunks; ++cc) r += __ldcg(p + cc * stride);
    double *o = job.out + (size_t)b0 * VD + tid;
    r *= sc;
    if (job.mode == OUT_ACCUMULATE) *o += r;
    else *o = r;
  }
  if (tid == 0) job.block_done[blk] = 0u;
}

template <int FD>
__global__ void __launch_bounds__(kChainBlock, 2) rpy_plain64_kernel(const QueueArgs q) {
  extern __shared__ __align__(16) double bb_smem[];
  __shared__ ChainShared sh;
  __shared__ int s_end[kQueueMaxJobs];
  __shared__ int s_unit, s_last;
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int j = 0; j < q.n_jobs; ++j) {
      const QueueJob &jb = q.jobs[j];
      const bool skip = jb.skip != nullptr && *jb.skip != 0;
      acc += skip ? 0 : (jb.n_tgt + kPlainTargets - 1) / kPlainTargets * jb.n_chunks;
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
    int lo = 0, hi = q.n_jobs - 1;  // first job whose end exceeds u
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_end[mid] > u) hi = mid; else lo = mid + 1;
    }
    const QueueJob &job = q.jobs[lo];
    const int local = u - (lo > 0 ? s_end[lo - 1] : 0);
    // the full chunks of all groups first, the short last ones at the end
    const int groups = (job.n_tgt + kPlainTargets - 1) / kPlainTargets;
    const int c = local / groups, grp = local - c * groups;
    if (job.vd == 6) plain_unit<6, FD>(job, grp, c, sh, bb_smem, &s_last);
    else plain_unit<3, FD>(job, grp, c, sh, bb_smem, &s_last);
    __syncthreads();  // s_unit and the shared buffers are reused by the next unit
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(q.counters + 1, 1u) == gridDim.x - 1) {
      q.counters[0] = 0u;
      q.counters[1] = 0u;
    }
  }
}

template <int FD>
static cudaError_t plain64_launch(const QueueArgs &a, long long units, cudaStream_t st) {
  constexpr int smem = 2 * 8 * chain_stage_elems<6, FD>(kPlainTargets);
  static std::atomic<int> occupancy[kMaxDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  int occ = occupancy[dev].load();
  if (occ == 0) {
    e = cudaFuncSetAttribute(rpy_plain64_kernel<FD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, rpy_plain64_kernel<FD>, kChainBlock, smem);
    if (e != cudaSuccess) return e;
    occupancy[dev].store(occ = occ < 1 ? 1 : occ);
  }
  const long long slots = (long long)occ * num_sms();
  rpy_plain64_kernel<FD><<<(int)std::min(units, slots), kChainBlock, smem, st>>>(a);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_plain64(int sources, const QueueJob *jobs, const QueueJob *jobs_host, int n_jobs,
                           unsigned *counters, cudaStream_t st, bool *taken) {
  *taken = false;
  if (sources == Q_SEG_BLOB) return cudaSuccess;
  long long units = 0;
  for (int j = 0; j < n_jobs; ++j) {
    const QueueJob &q = jobs_host[j];
    if (!q.plain) return cudaSuccess;
    units += (long long)((q.n_tgt + kPlainTargets - 1) / kPlainTargets) * q.n_chunks;
  }
  if (units == 0) return cudaSuccess;
  *taken = true;
  const QueueArgs a{jobs, n_jobs, counters};
  return sources == Q_SEG ? plain64_launch<6>(a, units, st) : plain64_launch<3>(a, units, st);
}

}  // namespace tfs
