// gfx_launch.cuh -- launches of the kernels that follow one another in a sweep or a check.
//
// On a small lattice a half-sweep lasts a few microseconds, and the gap between the end of a
// kernel and the start of the next is one of them.  launch_next() lets a kernel start when the
// blocks of the one before it in the stream have ended, before its writes have been made visible
// (programmatic dependent launch).  The rule for such a kernel: it begins with start_after(),
// which waits for those writes, touches no memory before, and reads what other kernels of the
// loop write with ordinary loads (ld_field).  A kernel launched otherwise, before or after, is
// ordered as always.  A half-sweep within a solve, before and after: FP32 4.0 -> 2.9 us on 8^4,
// 4.7 -> 3.9 on 16^4, 7.1 -> 6.3 on 16^3 x 32, 15.0 -> 14.1 on 24^4; FP64 7.3 -> 6.8 on 8^4,
// 19.4 -> 18.6 on 16^4.
// No kernel asks for the next one earlier (griddepcontrol.launch_dependents): its blocks then
// take the room that the running ones leave, which puts three on some SMs and one on others
// where a grid is less than a full wave (16^4 in FP64: 25.6 us).
#pragma once

#include <cuda_runtime.h>

namespace gfx {

__device__ __forceinline__ void start_after() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared,
                        cudaStream_t s, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = shared;
  c.stream = s;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace gfx
