// Launch settings of the sweep kernels: the opt-in to their shared memory, their
// resident blocks and the shared-memory carveout.  The runtime keeps a function's
// attributes per device, so they are found and set once per kernel and device.
#pragma once

#include <cuda_runtime_api.h>

#include <mutex>

namespace ouranos {

constexpr int kMaxDevices = 64;

// Shared-memory carveout for a launch on the current device `dev`: as much as the
// blocks that can be resident need, but at most what leaves keep_kb of the SM's
// on-chip memory to L1, where the cell-solve tables of the running directions live.
// The kernels that stream their sources element by element (cp.async.ca, which
// allocates in L1) keep 144 KB: fewer resident warps with their tables in L1
// beat more warps missing it (2-D Q2 S16 double-float sweep: 4 blocks per SM
// 1.63 ms, 3 blocks 1.40 ms, 2 blocks 1.35 ms); the 16-byte kernels (Q1 cells,
// cp.async.cg past L1) keep 32 KB (3-D Q1 GLC S12 FP32: 5 blocks 2.30 ms,
// 3 or 4 blocks 2.10 ms).
inline int carveout_percent(int dev, int grid, size_t smem_per_block, int max_blocks_per_sm, int keep_kb) {
  static std::mutex mu;
  static int sms[kMaxDevices] = {}, smem_sm[kMaxDevices] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (!sms[dev]) {
    cudaDeviceGetAttribute(&smem_sm[dev], cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  }
  if (sms[dev] < 1 || smem_sm[dev] < 1) return -1;  // leave the driver's choice
  const size_t per_block = smem_per_block + 1024;  // + the runtime's reserve per block
  int per_sm = (grid + sms[dev] - 1) / sms[dev];
  if (per_sm > max_blocks_per_sm) per_sm = max_blocks_per_sm;
  const long room = (long)smem_sm[dev] - (long)keep_kb * 1024;
  const int fit = room >= (long)per_block ? (int)(room / (long)per_block) : 1;
  if (per_sm > fit) per_sm = fit;
  const size_t need = (size_t)per_sm * per_block;
  const int pct = (int)((need * 100 + smem_sm[dev] - 1) / smem_sm[dev]);
  return pct < 100 ? pct : 100;
}

// One kernel's settings (a static object at its launch; zero: not set yet)
class SweepLaunch {
 public:
  // smem: dynamic shared memory of a block, smem_max: the most any launch of the
  // kernel asks for, smem_static: its static part; arrays: the source arrays of this
  // launch, 1 or 2, which smem goes by
  cudaError_t prepare(const void* kernel, int arrays, int grid, int block, size_t smem, size_t smem_max,
                      size_t smem_static, int keep_kb) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu_);
    PerDevice& d = dev_[dev];
    int& per_sm = d.per_sm[arrays - 1];
    if (!per_sm) {
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
      if (e != cudaSuccess) return e;
      int n = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, block, smem);
      if (e != cudaSuccess) return e;
      per_sm = n > 0 ? n : 1;
    }
    const int pct = carveout_percent(dev, grid, smem + smem_static, per_sm, keep_kb);
    if (pct >= 0 && pct + 1 != d.carve) {
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
      if (e != cudaSuccess) return e;
      d.carve = pct + 1;
    }
    return cudaSuccess;
  }

 private:
  struct PerDevice {
    int per_sm[2];  // resident blocks, by the number of source arrays
    int carve;      // last carveout asked for, plus one
  };
  std::mutex mu_;
  PerDevice dev_[kMaxDevices] = {};
};

}  // namespace ouranos
