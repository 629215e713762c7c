// What the tiled kernels need before they are launched on a device: more dynamic shared memory than
// the default 48 KB, and the number of blocks that are resident together, which their level chunks
// are chosen from.  Both belong to the device, so they are kept for each device, under a mutex.
#pragma once

#include <cuda_runtime_api.h>

#include <initializer_list>
#include <mutex>

namespace mgpu {

struct LaunchLimits {
  int occ = 0;  // resident blocks of an SM
  int nsm = 0;  // SMs of the device; 0: not set up yet
};

constexpr int LAUNCH_DEVICES = 64;
struct LaunchTable {
  std::mutex mu;
  LaunchLimits dev[LAUNCH_DEVICES];
};

// The limits on the current device for blocks of `threads` threads and `smem` bytes; the first call on
// a device sets the kernels up there.  The occupancy is that of the first kernel.  A kernel that cannot be set
// up leaves its error to the launch's check, and the next call tries again.
inline LaunchLimits launch_limits(LaunchTable& table, std::initializer_list<const void*> kernels, int threads,
                                  size_t smem) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  const bool kept = dev >= 0 && dev < LAUNCH_DEVICES;
  std::lock_guard<std::mutex> lock(table.mu);
  if (kept && table.dev[dev].nsm) return table.dev[dev];
  LaunchLimits l;
  bool ok = true;
  for (const void* k : kernels) {
    ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess && ok;
    ok = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess && ok;
  }
  ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&l.occ, *kernels.begin(), threads, smem) == cudaSuccess && ok;
  ok = cudaDeviceGetAttribute(&l.nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && ok;
  if (l.occ < 1) l.occ = 1;
  if (l.nsm < 1) l.nsm = 1;
  if (ok && kept) table.dev[dev] = l;
  return l;
}

}  // namespace mgpu
