// chain.cuh — kernels of a pass launched one behind the other on a stream
// (programmatic dependent launch): the next kernel's blocks start when those of
// the one before have ended, set up barriers and tensor memory, and wait until
// its results are visible, 1 to 3 us less for each kernel than an ordinary launch
// costs.  Us, ordinary / chained: LightSaber encapsulation, 17 instances 49.2 /
// 42.3; Saber, 4096: encapsulation 137 / 130, key generation 136 / 127,
// decapsulation with cached A 78 / 74; decapsulation 1: 59.9 / 57.9; FireSaber
// decapsulation 1000: 126 / 122.  (The next kernel's blocks let in while this
// one's still run, by griddepcontrol.launch_dependents: no better below 300
// instances, and up to 1.9 times as long above: they take the places over which
// the sponges of a Keccak launch are planned.)
//
// Every kernel launched by launch_chained calls chain_wait in all its threads
// before it touches global memory, so a kernel's completion implies that of all
// before it on the stream.  Launches of other kernels, copies and events order
// against these as always.
#pragma once
#include <cuda_runtime.h>

namespace tmvp {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <bool CHAINED = true, class... P, class... A>
inline cudaError_t launch_chained(void (*fn)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s,
                                  const A &...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = CHAINED ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

// Lets launches of fn ask for any dynamic shared memory that a block can have.
// The limit belongs to the kernel, for all host threads: one set to each launch's
// own size could refuse a larger launch that another thread is making.
template <class... P>
inline cudaError_t allow_shared_memory(void (*fn)(P...)) {
  constexpr int kBlockMax = 227 * 1024;
  cudaFuncAttributes at{};
  const cudaError_t e = cudaFuncGetAttributes(&at, fn);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kBlockMax - (int)at.sharedSizeBytes);
}

}  // namespace tmvp
