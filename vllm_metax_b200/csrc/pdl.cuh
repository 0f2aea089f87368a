// Programmatic dependent launch: a kernel may be started while the one before it in the stream drains, so that its launch, its
// barriers and its tensor memory are ready when that one ends.
//
// A kernel launched by pdl_run calls pdl_wait() in every thread before it touches anything that an earlier kernel may write or
// read - weights too, which a copy just before may have filled; a prefetch into L2, the point where all accesses meet, is the one
// thing that may come earlier.  Pointers in a file of such kernels carry no __restrict__: a load through a const one counts as a
// read of unchanging memory, which the compiler is free to move in front of the wait.  Only a launch that is captured into a graph right
// behind another kernel may start early: the wait covers kernels, and what else stands in front - small host-to-device copies, a
// memset, several nodes - has its ordinary order.
// pdl_trigger() lets the next kernel start as soon as every CTA of this one has got that far; it says nothing about results, for
// which the next one waits.  Without a dependent launch both do nothing.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether a launch into this stream may carry the attribute: it is being captured, and the one node in front is a kernel.
inline bool pdl_allowed(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess || status != cudaStreamCaptureStatusActive) return false;
  const cudaGraphNode_t* in_front = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n = 0;
  if (cudaStreamGetCaptureInfo_v3(stream, &status, nullptr, nullptr, &in_front, &edges, &n) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaGraphNodeType type = cudaGraphNodeTypeEmpty;
  return n == 1 && cudaGraphNodeGetType(in_front[0], &type) == cudaSuccess && type == cudaGraphNodeTypeKernel;
}

template <typename... P, typename... A>
inline cudaError_t pdl_run(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_allowed(stream) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace b200
