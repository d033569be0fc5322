// One warp waits on a barrier that nothing arrives at, and on one that has been
// arrived at: what tc::mbar_wait returns, and the time the first took.
#include <cuda_runtime.h>

#include "tc_sm100.cuh"

__global__ void wait_kernel(int* flag, int* ok, unsigned long long* ns) {
  __shared__ __align__(8) unsigned long long bar[2];
  const uint32_t b = so3g::tc::smem_u32(bar);
  if (threadIdx.x == 0) {
    so3g::tc::mbar_init(b, 1);
    so3g::tc::mbar_init(b + 8, 1);
    so3g::tc::mbar_fence_init();
    so3g::tc::mbar_arrive(b + 8);
  }
  __syncthreads();
  const bool here = so3g::tc::mbar_wait(b + 8, 0, flag, 1);
  const unsigned long long t = so3g::tc::global_ns();
  const bool never = so3g::tc::mbar_wait(b, 0, flag, 4);
  if (threadIdx.x == 0) ok[0] = here, ok[1] = never, *ns = so3g::tc::global_ns() - t;
}

extern "C" int run_wait(int* flag, int* ok, unsigned long long* ns) {
  int* d;
  if (cudaMalloc(&d, 64) != cudaSuccess || cudaMemset(d, 0, 64) != cudaSuccess) return 1;
  wait_kernel<<<1, 32>>>(d, d + 1, reinterpret_cast<unsigned long long*>(d + 4));
  int h[6];
  const cudaError_t e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(d);
  *flag = h[0], ok[0] = h[1], ok[1] = h[2];
  *ns = *reinterpret_cast<unsigned long long*>(h + 4);
  return e != cudaSuccess;
}
