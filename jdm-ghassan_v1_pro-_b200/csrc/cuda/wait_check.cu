// The bounded waits of the tensor-core kernels (sm100_common.cuh), run until they give up: see gb_wait_check in gb_api.h.
#include "sm100_common.cuh"
#include "gb_api.h"

namespace gb {

__global__ void __launch_bounds__(96) wait_check_kernel(int waits, long long limit, long long* out, int* status) {
  __shared__ uint64_t empty_bar, full_bar;
  __shared__ int abort_word, issued;
  volatile int* abort_flag = &abort_word;
  if (threadIdx.x == 0) {
    mbar_init(&empty_bar, 1);
    mbar_init(&full_bar, 1);
    abort_word = 0;
    issued = 0;
    fence_barrier_init();
  }
  __syncthreads();
  const long long t0 = clock64();
  if (threadIdx.x < 32) {
    const uint32_t on = elect_one();
    for (int i = 0; i < waits; ++i) {
      wait_or_leave(&empty_bar, 0, status, ST_TIMEOUT_EMPTY, abort_flag, limit);
      if (on) ++issued;
    }
    __syncwarp();
  } else if (threadIdx.x < 64) {
    for (int i = 0; i < waits; ++i) wait_or_report(&full_bar, 0, status, ST_TIMEOUT_FULL, abort_flag, limit);
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x == 64) { out[0] = clock64() - t0; out[1] = issued; }      // the first warp's threads have ended
}

}  // namespace gb

extern "C" int gb_wait_check(int waits, long long limit, long long* out, int* status, cudaStream_t stream) {
  if (waits < 1 || waits > 1000 || limit < 1 || limit > gb::WAIT_CYCLES || !out || !status) return -1;
  gb::wait_check_kernel<<<1, 96, 0, stream>>>(waits, limit, out, status);
  return gb_launch_rc();
}
