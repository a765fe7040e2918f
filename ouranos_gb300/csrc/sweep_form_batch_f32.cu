// The batched launch of the default forms in FP32 (sweep_lane.cuh, sweep_group.cuh).
#include "sweep_lane.cuh"

namespace ouranos {
template <int DIM>
static cudaError_t form_batch(int p1, int fm, int lpc, const BatchLaunch<float>& b, cudaStream_t s) {
  return lpc == 1 ? launch_lane_batch_dim<float, DIM>(p1, fm, b, s) : launch_group_batch_dim<float, DIM>(p1, fm, lpc, b, s);
}
template <>
cudaError_t launch_sweep_form_batch<float, 2>(int p1, int fm, int lpc, bool sources, const SweepArgs<float>* args,
                                           const int2* tmap, int n_total, int* ticket, const int* status,
                                           const unsigned* epoch, int grid, int block, cudaStream_t s) {
  return form_batch<2>(p1, fm, lpc, {args, tmap, n_total, ticket, status, epoch, sources, grid, block}, s);
}
template <>
cudaError_t launch_sweep_form_batch<float, 3>(int p1, int fm, int lpc, bool sources, const SweepArgs<float>* args,
                                           const int2* tmap, int n_total, int* ticket, const int* status,
                                           const unsigned* epoch, int grid, int block, cudaStream_t s) {
  return form_batch<3>(p1, fm, lpc, {args, tmap, n_total, ticket, status, epoch, sources, grid, block}, s);
}
}  // namespace ouranos
