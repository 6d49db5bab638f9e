// Launches that are programmatic dependents of one another: a kernel is launched
// while the one before it runs, and waits for its end in wait_for_previous().  The
// kernels of a small network's step take 1.5 to 8 us each, up to 1 us of it (4 us
// where the step is not in a graph) the way from one's end to the next one's start.
// A step of the 784-500-10 classifier 57 -> 48 us, of the 256 x 256 spnet network
// 116 -> 99 us, of the 32 x 32 Izhikevich network (a graph) 21.8 -> 21.3 us.
#pragma once
#include <utility>

#include "cuda_check.h"

namespace sg {

// Waits for the kernel before, whose writes are then visible, and lets the one after
// be launched.  First in every kernel that launch_dependent starts, by every thread:
// a kernel that ended without it could be followed by one that overtakes the kernel
// before both.  Nothing happens in a launch of another kind.
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// p for loads after the wait that the compiler is not to move before it (read-only
// ones, which no memory clobber holds), in kernels that load anything before it.
// What may be loaded before it is what the kernel before does not write: the one
// before that has completed, its writes included, since the kernel before waited for
// it before it let this one be launched.  So a kernel may load early what another one
// writes only if a kernel that waits stands between the two in its stream, or an event
// wait followed by such a kernel where the other one runs in another stream.  Nothing
// checks that: Engine::enqueue_step says where its order provides it.
template <class T>
__device__ __forceinline__ T* after_wait(T* p) {
    asm volatile("" : "+l"(p));
    return p;
}

// SMs of the device, for rules on how many CTAs it holds.
inline int num_sms() {
    static const int sms = [] {
        int dev = 0, n = 0;
        SG_CUDA(cudaGetDevice(&dev));
        SG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        return n;
    }();
    return sms;
}

template <class... P, class... A>
void launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                      A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...));
}

}  // namespace sg
