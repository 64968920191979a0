// Programmatic dependent launches: a kernel launched with launch_dependent()
// may become resident while its predecessor in the stream drains, so its
// launch and its prologue (twiddle tables, barrier set-up, parameters) hide
// behind the predecessor's last blocks.
//
// Contract of such a kernel: every thread of every block (but those of blocks
// that leave at once) calls depend_wait() before it touches memory that an
// earlier kernel of the stream writes, or writes memory that one reads, and
// depend_trigger(), if at all, only after it.  depend_wait() returns when the
// predecessor has completed and its writes are visible; as the predecessor
// waited in the same way, so have all before it.  Before depend_wait() a
// kernel may read what was complete when the chain began: a block can only run
// once all blocks of its predecessor have triggered or ended, that is have
// seen their own predecessor complete.  What it reads after the wait goes
// through after_wait() pointers.  Behind a copy the launch is an ordinary one.
//
// A block that ends triggers.  An earlier depend_trigger() lets the successor's
// blocks in as soon as this kernel's have all started: worth it for launches
// of a few blocks with long prologues (the streamed engine: a step of one
// 128^2 world of 3 channels x 15 kernels 25 -> 19 us), not where a last partial
// wave still needs the SMs evenly (the N-D engine: 8 steps of 2 worlds of
// 1024^2, 646 us as ordinary launches, 662 with early triggers, 603 without).
#pragma once
#include <cuda_runtime.h>

namespace lgx {

__device__ __forceinline__ void depend_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void depend_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The pointer as it is after depend_wait(): loads through it stay behind the
// wait even where the compiler takes the memory for constant (const
// __restrict__, __ldg).
template <class T>
__device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace lgx
