// The sweep with one lane to a cell in double-float (sweep_lane.cuh).
#include "sweep_lane.cuh"

namespace ouranos {
template <>
cudaError_t launch_sweep_lane<df64, 2>(int p1, int fm, const SweepArgs<df64>& a, int grid, int block, cudaStream_t s) {
  return launch_lane_dim<df64, 2>(p1, fm, a, grid, block, s);
}
template <>
cudaError_t launch_sweep_lane<df64, 3>(int p1, int fm, const SweepArgs<df64>& a, int grid, int block, cudaStream_t s) {
  return launch_lane_dim<df64, 3>(p1, fm, a, grid, block, s);
}
}  // namespace ouranos
