// pdl.cuh -- device side of programmatic dependent launches.
#pragma once
#include <cuda_runtime.h>

namespace dnsb {

// A kernel launched by launch_pdl (launch.h) takes as its last argument
// whether it is a programmatic dependent of the stream's previous kernel.
//
// pdl_wait returns once every grid this one depends on has finished and its
// writes are visible.  Every block executes it before its first access to
// memory that another kernel writes or reads, so a chain of dependent
// launches keeps stream order.  What another kernel of the stream writes is
// read through plain pointers: __ldg and const __restrict__ allow the compiler
// to move a load above the wait, and so does a __restrict__ pointer that the
// kernel also writes through (the compiler may take the wait's assembly not to
// touch what it points to).  __restrict__ is for the context's tables, which no
// kernel of a step writes, and for outputs that are only written, from values
// loaded past the wait (tests/test_dependent_launches.py lists both).
__device__ __forceinline__ void pdl_wait(int dep) {
  if (dep) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Lets the dependent grid become resident in the slots this grid leaves free
// (it takes effect once every block has executed it or exited, so it never
// displaces a block of this grid).
__device__ __forceinline__ void pdl_trigger(int dep) {
  if (dep) asm volatile("griddepcontrol.launch_dependents;");
}

}  // namespace dnsb
