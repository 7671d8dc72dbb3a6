// Programmatic dependent launch, device side.
//
// A kernel launched with the programmatic stream serialization attribute is set up while the stream's
// previous kernel ends, so its first instructions may run before that kernel's stores are visible.
// griddepcontrol.wait is what orders them, and it orders loads only as far as the compiler keeps them
// behind it: it may move a load that it takes for read-only (through a const __restrict__ parameter,
// __ldg, ld.global.nc, asm without volatile) to any place where the address is known.
// wait_for_previous therefore takes the pointers through which the kernel reads what the previous one
// may write, and gives them back as values that the compiler knows nothing about before the wait: a
// load through them cannot come earlier and is no longer taken for read-only.  For the same reason
// none of these loads is an .nc one, whose data must not change while the kernel is resident.
//
// What kernels before the previous one wrote is complete when a kernel starts (the previous one's
// blocks have all passed their own wait by then, or it was launched without the attribute), so within
// a chain only the previous kernel's output is passed, and the rest is read as ever.  (With every input
// passed, and the walk waiting too, a step of 1M particles takes 1,154 us against 1,129: the walk's
// loads then keep their place among the warp barriers.)  Without the launch attribute the wait does
// nothing.
#pragma once

#include <cuda_runtime.h>

namespace akua {
namespace pdl {

// `p` (global memory) as a new value, still known to point to global memory.
template <class P>
__device__ __forceinline__ void renew(P& p) {
    size_t a = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(a));
    p = (P)__cvta_global_to_generic(a);
}

template <class... P>
__device__ __forceinline__ void wait_for_previous(P&... read) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (renew(read), ...);
}

}  // namespace pdl
}  // namespace akua
