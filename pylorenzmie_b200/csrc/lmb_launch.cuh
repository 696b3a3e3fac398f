// Launch helpers shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "lmb200.h"

#define LMB_CK(x)                                    \
  do {                                               \
    cudaError_t e_ = (x);                            \
    if (e_ != cudaSuccess) return LMB_ERR_CUDA;      \
  } while (0)

namespace lmb {

// Per-call host work kept off the path between fits: the shared-memory
// attribute of a kernel is raised once per device to the largest size asked
// for, and persistent grid sizes are looked up once per (device, kernel,
// block, shared memory).
inline std::mutex g_launch_cache_lock;
struct AttrEntry {
  int device;
  const void* fn;
  size_t value;
  int tpb;
  size_t smem;
};
inline std::vector<AttrEntry> g_smem_set;    // value: bytes set
inline std::vector<AttrEntry> g_grid_sizes;  // value: grid

// Whether npts is the grid's number of pixels.
inline bool grid_holds(const lmb_grid* grid, long long npts) {
  if (grid->nx < 1 || grid->ny < 1) return npts == 0;
  return npts / grid->nx == grid->ny && npts % grid->nx == 0;
}

inline int current_device() {
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

inline cudaError_t smem_attr(const void* fn, size_t bytes) {
  // A launch may use 48 KB without the attribute, its static shared memory
  // included (the kernels here declare less than 4 KB).
  if (bytes <= 44 * 1024) return cudaSuccess;
  const int dev = current_device();
  std::lock_guard<std::mutex> hold(g_launch_cache_lock);
  for (const AttrEntry& e : g_smem_set)
    if (e.device == dev && e.fn == fn && e.value >= bytes) return cudaSuccess;
  const cudaError_t r = cudaFuncSetAttribute(
      fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  if (r != cudaSuccess || dev < 0) return r;
  for (AttrEntry& e : g_smem_set)
    if (e.device == dev && e.fn == fn) {
      e.value = bytes;
      return r;
    }
  g_smem_set.push_back({dev, fn, bytes, 0, 0});
  return r;
}

}  // namespace lmb
