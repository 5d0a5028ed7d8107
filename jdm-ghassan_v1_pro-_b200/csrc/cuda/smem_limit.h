// How much dynamic shared memory a kernel may be launched with.
#pragma once
#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <utility>

// More than 48 KB of static and dynamic shared memory together want a limit of the kernel raised: asked for from 16 KB of dynamic memory on, since no kernel
// here has more than 32 KB of static.  (Asked for above 48 KB of dynamic memory, launches just below, 2 x 4096 numbers and two norms in layers_gemv.cu, were refused.)  The limit of a kernel on a device only ever grows, under a lock: a thread whose launch
// needs less must not take it back between another thread's raising it and that thread's launch.  0, or -10.
inline int gb_allow_smem(const void* kernel, size_t bytes) {
  if (bytes <= 16 * 1024) return 0;
  static std::mutex lock;
  static std::map<std::pair<const void*, int>, size_t> limits;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return -10; }
  try {
    const std::lock_guard<std::mutex> held(lock);
    size_t& limit = limits[{kernel, dev}];
    if (bytes > limit) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) { (void)cudaGetLastError(); return -10; }
      limit = bytes;
    }
  } catch (...) {                                       // no memory for the table's entry
    return -10;
  }
  return 0;
}
