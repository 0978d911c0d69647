// Device side of chained launches (launch_tiles, ssd_host.h).  Every kernel calls both, in every thread (the first returns at once in a kernel
// launched without chaining):
//
//   after_previous()  before any access to global memory: returns when the kernel before it in the stream has finished and its
//                     writes are visible.  Each kernel waits itself, so that its end implies the end of all before it.
//   allow_next()      lets the next kernel's CTAs be placed once every CTA of this one got here.  After the wait above, and
//                     after this CTA has its tensor memory: a waiting CTA of the next kernel may hold tensor memory, and one of
//                     this kernel must never have to wait for that.
#pragma once

namespace ssd {

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace ssd
