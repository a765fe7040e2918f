// The sweep with several lanes to a cell in FP32, 3-D (sweep_group.cuh).
#include "sweep_group.cuh"

namespace ouranos {
template <>
cudaError_t launch_sweep_group<float, 3>(int p1, int fm, const SweepArgs<float>& a, int grid, int block, cudaStream_t s) {
  return launch_group_dim<float, 3>(p1, fm, a, grid, block, s);
}
}  // namespace ouranos
