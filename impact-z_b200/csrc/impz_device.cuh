// impz_device.cuh -- device helpers shared by the kernel headers.
#pragma once
#include <cuda_runtime.h>

namespace impz {

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization (launch_pdl) may be scheduled while the previous kernel on
// its stream drains; it waits here, before reading anything that kernel
// wrote.  For an ordinary launch this returns at once.
__device__ __forceinline__ void griddep_wait() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// Lets the next kernel of the stream be scheduled as soon as every block of
// this one has called it.  Worth it for kernels that are little more than
// their launch; in the step's chain of kernels it cost more than it hid (the
// early blocks of the next transform held the shared memory that the
// running one's blocks wanted: 22 -> 27 us for the convolution of 32x32x64).
__device__ __forceinline__ void griddep_launch() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

// Brings the 128-byte line at p into L2, without waiting and without a register.
__device__ __forceinline__ void prefetch_l2(const void* p) {
#if defined(__CUDA_ARCH__)
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
#endif
}

}  // namespace impz
