// The sweep with several lanes to a cell in FP64, 3-D (sweep_group.cuh).
#include "sweep_group.cuh"

namespace ouranos {
template <>
cudaError_t launch_sweep_group<double, 3>(int p1, int fm, const SweepArgs<double>& a, int grid, int block, cudaStream_t s) {
  return launch_group_dim<double, 3>(p1, fm, a, grid, block, s);
}
}  // namespace ouranos
