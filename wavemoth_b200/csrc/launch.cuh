// Launches of kernels that overlap their start with the end of the kernel
// before them (programmatic dependent launch).
//
// The kernels of one transform follow each other on one stream, and for small
// transforms each is hardly longer than the gap that a plain launch leaves plus
// its own chain of table look-ups.  A kernel launched here may start when the
// CTAs of the kernel before it have exited, before that kernel counts as
// complete; it reads its plan's tables, which no kernel of a call writes, and
// waits (grid_wait) for the complete kernels before it, and their memory, ahead
// of its first access to anything else.  Every CTA calls grid_wait, so a kernel
// that has completed implies that all before it have.
//
// Measured, us, plain -> overlapped: map2alm of 3 maps at nside 32 16.2 ->
// 13.7, alm2map of 1 map at nside 64 20.5 -> 15.9, three iterations of 3 maps at
// nside 128 255 -> 223.  Letting the next kernel start earlier still (a trigger
// at a kernel's top or before its last stores) made the iterations slower (264,
// 236): its CTAs settle where the first SMs fall idle.
#pragma once
#include <cuda_runtime.h>

namespace wm {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Plain launches while the stream is captured: a graph's branches join at
// kernels that depend on several others.
template <class... Params, class... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t st,
                              const Args &...args) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  const bool known = cudaStreamIsCapturing(st, &capture) == cudaSuccess;
  if (!known) cudaGetLastError();
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((unsigned)grid);
  config.blockDim = dim3((unsigned)block);
  config.dynamicSmemBytes = smem;
  config.stream = st;
  config.attrs = &overlap;
  config.numAttrs = known && capture == cudaStreamCaptureStatusNone ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

}  // namespace wm
