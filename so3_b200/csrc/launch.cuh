// Launches that overlap their start with the end of the kernel before them
// (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

#include "so3gpu_internal.h"

namespace so3g {

// Device side: dep_launch lets the next kernel's CTAs become resident once
// every CTA of this one has come to it; dep_wait waits until the kernel before
// has finished and its writes are visible.  Nothing a kernel of the stream
// writes may be touched before dep_wait; tables built ahead of the transforms
// may.  dep_launch stands where a CTA has its inputs or its results, not at the
// start: CTAs that become resident early pile up on the SMs that have room and
// then share them (L = 64, N = 8: 61.5 us without, 66.3 at the start, 51.0 late).
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Host side.  A transform is four launches of a few microseconds at small band
// limits; the start of each (CTA launch, parameters, first table reads) hides
// behind the one before.  Inverse + forward (us): L = 16, N = 4 36.9 -> 24.8, L =
// 32, N = 8 45 -> 31, L = 64, N = 64 156 -> 137, L = 256, N = 16 733 -> 717.
// Captured streams take plain launches.
template <class... P, class... A>
int launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  if (int rc = allow_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const bool plain = cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = plain ? 0 : 1;
  SO3G_CUDA(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...));
  SO3G_LAUNCHED();
  return kOk;
}

}  // namespace so3g
