// Self-test of the bounded wait every role of the attention kernel uses (wait_bar and give_up, common.cuh): three warps wait, one with
// a SHORT poll limit, the others with the limits that the roles have, on an mbarrier phase that nothing will ever complete, each
// behind a wait for a phase that counts as complete.  Those for the former must run out, record their code in the status word and let the kernel return normally - no trap, no fault, no
// hang - which is how a protocol error inside the attention kernel surfaces as SAGE3_ERR_DEVICE_WAIT on the host.  No
// counterpart in the reference (its kernel waits without bounds).
#include "common.cuh"
#include "kernels.h"

namespace sage3 {

namespace {

__global__ void __launch_bounds__(96) bounded_wait_selftest_kernel(int* status) {
  __shared__ __align__(8) unsigned long long bar_mem;
  __shared__ int abort_flag;
  const uint32_t bar = smem_u32(&bar_mem);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(bar, 1);                  // one arrival expected, none will come
    fence_mbar_init();
  }
  __syncthreads();
  const int warp = threadIdx.x / 32;
  // (parity 1 counts as complete on a fresh barrier; 2048 polls of 4 us at most: gives up after a few milliseconds)
  int fail = warp == 0 ? wait_bar<76, 2048>(bar, 1) : wait_bar_uniform<75>(bar, 1);
  if (fail == 0) fail = warp == 0 ? wait_bar<77, 2048>(bar, 0) : (warp == 1 ? wait_bar<78>(bar, 0) : wait_bar_uniform<79>(bar, 0));
  if (fail != 0) give_up(&abort_flag, status, fail);
  else atomicCAS(status, 0, -1);        // cannot happen; would mean the wait saw a phase nobody completed
}

}  // namespace

cudaError_t launch_bounded_wait_selftest(int* status, cudaStream_t stream) {
  bounded_wait_selftest_kernel<<<1, 96, 0, stream>>>(status);
  return cudaGetLastError();
}

}  // namespace sage3
