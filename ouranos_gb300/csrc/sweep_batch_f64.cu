// Instantiations of the batched sweep kernel in double: 2-D Q1 and Q2,
// 3-D Q1 per lane; the default forms come from sweep_form_batch_f64.cu.
#include "sweep.cuh"

namespace ouranos {

template <>
cudaError_t launch_sweep_batch<double>(int dim, int p1, int fm, int lpc, bool grouped, bool sources,
                                   const SweepArgs<double>* args, const int2* tmap,
                                   int n_total, int* ticket, const int* status, const unsigned* epoch,
                                   int grid, int block, cudaStream_t s) {
  if (grouped)
    return dim == 2 ? launch_sweep_form_batch<double, 2>(p1, fm, lpc, sources, args, tmap, n_total, ticket, status, epoch, grid, block, s)
                    : launch_sweep_form_batch<double, 3>(p1, fm, lpc, sources, args, tmap, n_total, ticket, status, epoch, grid, block, s);
#define ARGS fm, lpc, args, tmap, n_total, ticket, status, epoch, grid, block, s
  if (dim == 2) {
    switch (p1) {
      case 2: return launch_sweep_batch_impl<double, 2, 2>(ARGS);
      case 3: return launch_sweep_batch_impl<double, 2, 3>(ARGS);
    }
  } else if (dim == 3) {
    switch (p1) {
      case 2: return launch_sweep_batch_impl<double, 3, 2>(ARGS);
    }
  }
#undef ARGS
  return cudaErrorInvalidValue;
}

}  // namespace ouranos
