// Instantiations of the sweep kernel in double-float (FP64 accuracy on the
// FP32 pipes): the per-lane forms of the explicit tilings, 2-D Q1 and Q2, 3-D Q1
// (the default forms: sweep_lane_df64.cu, sweep_group_df64_*.cu; one warp per
// cell: sweep_wide_df64.cu).
#include "sweep.cuh"

namespace ouranos {

template <>
cudaError_t launch_sweep<df64>(int dim, int p1, int fm, const SweepArgs<df64>& a, int grid, int block,
                               cudaStream_t s) {
  if (a.grouped && a.lpc == 1)
    return dim == 2 ? launch_sweep_lane<df64, 2>(p1, fm, a, grid, block, s)
                    : launch_sweep_lane<df64, 3>(p1, fm, a, grid, block, s);
  if (a.grouped)
    return dim == 2 ? launch_sweep_group<df64, 2>(p1, fm, a, grid, block, s)
                    : launch_sweep_group<df64, 3>(p1, fm, a, grid, block, s);
  if (a.lpc == 32) return launch_sweep_wide<df64>(dim, p1, a, grid, block, s);
  if (dim == 2) {
    switch (p1) {
      case 2: return launch_sweep_impl<df64, 2, 2>(fm, a, grid, block, s);
      case 3: return launch_sweep_impl<df64, 2, 3>(fm, a, grid, block, s);
    }
  } else if (dim == 3) {
    switch (p1) {
      case 2: return launch_sweep_impl<df64, 3, 2>(fm, a, grid, block, s);
    }
  }
  return cudaErrorInvalidValue;
}

}  // namespace ouranos
