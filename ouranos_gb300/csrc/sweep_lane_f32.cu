// The sweep with one lane to a cell in FP32 (sweep_lane.cuh).
#include "sweep_lane.cuh"

namespace ouranos {
template <>
cudaError_t launch_sweep_lane<float, 2>(int p1, int fm, const SweepArgs<float>& a, int grid, int block, cudaStream_t s) {
  return launch_lane_dim<float, 2>(p1, fm, a, grid, block, s);
}
template <>
cudaError_t launch_sweep_lane<float, 3>(int p1, int fm, const SweepArgs<float>& a, int grid, int block, cudaStream_t s) {
  return launch_lane_dim<float, 3>(p1, fm, a, grid, block, s);
}
}  // namespace ouranos
