// Instantiations of the sweep kernel in double: the per-lane forms of the
// explicit tilings, 2-D Q1 and Q2, 3-D Q1 (the default forms: sweep_lane_f64.cu,
// sweep_group_f64_*.cu; one warp per cell: sweep_wide_f64.cu).
#include "sweep.cuh"

namespace ouranos {

template <>
cudaError_t launch_sweep<double>(int dim, int p1, int fm, const SweepArgs<double>& a, int grid, int block,
                                cudaStream_t s) {
  if (a.grouped && a.lpc == 1)
    return dim == 2 ? launch_sweep_lane<double, 2>(p1, fm, a, grid, block, s)
                    : launch_sweep_lane<double, 3>(p1, fm, a, grid, block, s);
  if (a.grouped)
    return dim == 2 ? launch_sweep_group<double, 2>(p1, fm, a, grid, block, s)
                    : launch_sweep_group<double, 3>(p1, fm, a, grid, block, s);
  if (a.lpc == 32) return launch_sweep_wide<double>(dim, p1, a, grid, block, s);
  if (dim == 2) {
    switch (p1) {
      case 2: return launch_sweep_impl<double, 2, 2>(fm, a, grid, block, s);
      case 3: return launch_sweep_impl<double, 2, 3>(fm, a, grid, block, s);
    }
  } else if (dim == 3) {
    switch (p1) {
      case 2: return launch_sweep_impl<double, 3, 2>(fm, a, grid, block, s);
    }
  }
  return cudaErrorInvalidValue;
}

}  // namespace ouranos
