// rpy_queue_f32.cu -- FP32 (compensated) instantiations of the work-queue
// kernel: (threads per CTA, targets per thread, sources per tile, minimum
// resident CTAs); index = variant.
#include "rpy_queue.cuh"

namespace tfs {

const QueueVariant g_qvariants_f32[kNumQueueVariantsF32] = {
    {128, 1, 256, 5}, {128, 2, 256, 3}, {64, 1, 256, 10}, {64, 2, 256, 6}, {128, 4, 256, 2}};

const QueueFn g_queue_f32[kNumQueueVariantsF32][kNumQueueSources] = {
    TFS_QUEUE_ROW(float, 128, 1, 256, 5), TFS_QUEUE_ROW(float, 128, 2, 256, 3),
    TFS_QUEUE_ROW(float, 64, 1, 256, 10), TFS_QUEUE_ROW(float, 64, 2, 256, 6),
    TFS_QUEUE_ROW(float, 128, 4, 256, 2)};

// The plain form (segment or blob sources alone).
const QueueVariant g_qvariant_f32_plain = {128, 1, 256, 8};
const QueueFn g_queue_f32_plain[kNumQueueSources] = {
    queue_launch_fn<float, 6, 0, 128, 1, 256, 8, false>,
    queue_launch_fn<float, 3, 0, 128, 1, 256, 8, false>, nullptr};

}  // namespace tfs
