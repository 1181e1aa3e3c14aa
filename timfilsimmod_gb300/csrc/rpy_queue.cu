// rpy_queue.cu -- host side of the work-queue products (rpy_queue.cuh):
// source chunking, grid sizing and the launch.
#include <cuda_runtime.h>

#include <algorithm>

#include "tfs_kernels.h"

namespace tfs {

// Units of 128 targets that a product is cut into where there is work enough,
// and about as many as a GB300 runs at once (152 SMs of four to five CTAs).
// Constants, not the launch's own occupancy: the chunks fix the order of the sums,
// and a product's bits depend on its sizes alone, not on the variant that runs it.
constexpr long kUnits = 8192, kQueueFill = 700;

void queue_chunking(int n_src, int n_particles, int *chunk, int *n_chunks) {
  if (n_src <= 0) {
    *chunk = kQueueQuantum;
    *n_chunks = 0;
    return;
  }
  const long blocks = std::max(1L, ((long)n_particles + 127) / 128);
  const long want = std::max(1L, std::min<long>(kMaxSplits, (kUnits + blocks - 1) / blocks));
  long c = ((long)n_src + want - 1) / want;
  c = ((c + kQueueQuantum - 1) / kQueueQuantum) * kQueueQuantum;
  *chunk = (int)c;
  *n_chunks = (int)(((long)n_src + c - 1) / c);
}

// Where 256-source chunks would give fewer units than run at once, smaller ones
// (M_ss of 640 segments, 15 and 100 units: 61 and 37 us; M_bb of 2 562 blobs,
// 231 and 567: 41 and 29 us); elsewhere 256, as a unit's own cost (target and
// source loads, partial sums, its turn at the counters) is about 5 us (M_sb of
// 2 562 blobs on 12 800 segments, 1 100 and 4 100 units: 56 and 80 us).
void queue_chunking32(int n_src, int n_tgt, int *chunk, int *n_chunks) {
  if (n_src <= 0) {
    *chunk = kQueueQuantum32;
    *n_chunks = 0;
    return;
  }
  const long blocks = std::max(1L, ((long)n_tgt + 127) / 128);
  long want;
  if (blocks * (((long)n_src + 255) / 256) < kQueueFill)
    want = kQueueFill / blocks;  // as many units as run at once
  else
    want = (kUnits + blocks - 1) / blocks;
  want = std::max(1L, std::min<long>(kMaxSplits, want));
  long c = ((long)n_src + want - 1) / want;
  const long quantum = c < 256 ? kQueueQuantum32 : 256;
  c = ((c + quantum - 1) / quantum) * quantum;
  if (blocks * (((long)n_src + 255) / 256) >= kQueueFill) c = std::max(c, 256L);
  *chunk = (int)c;
  *n_chunks = (int)(((long)n_src + c - 1) / c);
}

long long queue_units(const QueueJob *jobs_host, int n_jobs, int block_targets) {
  long long u = 0;
  for (int j = 0; j < n_jobs; ++j)
    u += (long long)((jobs_host[j].n_tgt + block_targets - 1) / block_targets) *
         (jobs_host[j].plain ? jobs_host[j].n_chunks : jobs_host[j].n_chunks32);
  return u;
}

cudaError_t launch_queue(int fp32, int variant, int sources, const QueueJob *jobs,
                         const QueueJob *jobs_host, int n_jobs, unsigned *counters,
                         cudaStream_t st, cudaEvent_t *ev) {
  if (sources < 0 || sources >= kNumQueueSources || n_jobs < 0 || n_jobs > kQueueMaxJobs)
    return cudaErrorInvalidValue;
  const int nvar = fp32 ? kNumQueueVariantsF32 : kNumQueueVariantsF64;
  if (variant < 0 || variant >= nvar) variant = 0;
  if (!fp32) {
    if (ev) cudaEventRecord(ev[0], st);
    bool taken = false;  // (a pinned variant keeps the tile form)
    cudaError_t e = cudaSuccess;
    if (variant == 0) e = launch_plain64(sources, jobs, jobs_host, n_jobs, counters, st, &taken);
    if (e == cudaSuccess && !taken)
      e = launch_fx(variant, sources, jobs, jobs_host, n_jobs, counters, st);
    if (ev) cudaEventRecord(ev[1], st);
    return e;
  }
  const bool plain = n_jobs > 0 && jobs_host[0].plain != 0;
  const QueueVariant var = plain ? g_qvariant_f32_plain : g_qvariants_f32[variant];
  const QueueFn fn = plain ? g_queue_f32_plain[sources] : g_queue_f32[variant][sources];
  if (fn == nullptr) return cudaErrorInvalidValue;
  const long long units = queue_units(jobs_host, n_jobs, var.block * var.tpt);
  if (units <= 0) return cudaSuccess;
  int resident = 1;
  cudaError_t e = fn(QueueArgs{}, 0, st, &resident);
  if (e != cudaSuccess) return e;
  const long long slots = (long long)resident * num_sms();
  const int ctas = (int)std::min(slots, units);
  if (ev) cudaEventRecord(ev[0], st);
  e = fn(QueueArgs{jobs, n_jobs, counters}, ctas, st, nullptr);
  count_launch();
  if (ev) cudaEventRecord(ev[1], st);
  return e;
}

}  // namespace tfs
