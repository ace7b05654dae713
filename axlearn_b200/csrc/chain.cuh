// Chained launches of a decoding step: each kernel of the chain is put on the GPU while its predecessor still runs
// (programmatic dependent launch), so that a launch, a prologue and -- in the weight-streaming GEMM -- the first tiles
// of weights are no longer paid one after the other.
//
// A kernel of the chain calls `chain_link()` first: it lets its successor start and then waits until everything before
// it has finished and is visible.  All threads call it, ahead of any early return: a successor that waits for this
// kernel thereby waits for all kernels before it, too.  Launched in the ordinary way both instructions do nothing.
//
// What earlier kernels write (activations, lengths, partial results, copies of parameters) is read with ordinary loads,
// through pointers without `__restrict__`, and never with `__ldg`: the read-only path is promised for data that is
// constant while the kernel is resident, which a chained kernel is before its input is written, and no wait orders it.
// Only tables of parameters that a step does not write may be `const __restrict__`.
//
// Launches are chained only while the calling thread captures a decoding step (`axb_chain_launches`): there, what may
// be read ahead of the wait is known.  Kernels that stream much memory in one wave or with many small CTAs (expert
// products, state-space and latent decoding) keep ordinary launches: started early, their CTAs go to the SMs that
// happen to have room, and the uneven spread costs more than the launch (32 experts at batch 16: 59 -> 92 us, state-space
// decoding 21.5 -> 25).
//
// Captured steps, separate / chained launches (us a step, best of 12 replays): 1B widths, 4 layers, batch 1: 326 / 280;
// 8B widths, 4 layers, batch 16: 766 / 720; Zukitar 1B widths, 3 layers: batch 1 263 / 243, batch 16 380 / 354.
#pragma once

#include <cuda_runtime.h>

namespace axb {

inline thread_local bool chain_launches = false;

__device__ __forceinline__ void chain_start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_link() {
  chain_start_next();
  chain_wait();
}

// Adds the attribute of a chained launch to `attr` when launches are chained; returns the number of attributes.
inline int chain_attribute(cudaLaunchAttribute* attr, int count) {
  if (!chain_launches) return count;
  attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[count].val.programmaticStreamSerializationAllowed = 1;
  return count + 1;
}

template <typename... Params, typename... Args>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                           Args&&... args) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = static_cast<unsigned>(chain_attribute(attr, 0));
  cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);  // errors: cudaGetLastError, as after <<< >>>
}

}  // namespace axb
