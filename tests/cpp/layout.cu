// Shared memory of the kernels' work buffers, their static part included, for tests/test_layout.py.
#define MQ_DEVICE_ONLY
#include "walker_kernels.cuh"

extern "C" long layout_bytes(int kind, int L, int maxA, int maxB, int G) {
  const int pa = mq::padld(maxA > maxB ? maxA : maxB), pb = mq::padld(maxB), pq = mq::padld(2 * maxB);
  const long fixed = mq::kOpBytes;
  switch (kind) {
    case 0:  // the engine's FP64 kernels
      return fixed + 8 * mq::smem_doubles(L, maxA, maxB, G, pa, pb, pq, nullptr, nullptr);
    case 1:  // the per-walker TF32 sweep
      return fixed + mq::smem_bytes_f32(L, maxA, maxB, G, pa, pb, nullptr, nullptr);
    default:  // the allocation-free local energy
      return fixed + 8 * mq::smem_doubles(L, maxA, maxB, 1, pa, pb, pq, nullptr, nullptr, nullptr, nullptr, false, false);
  }
}
