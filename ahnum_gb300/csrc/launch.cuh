// Launch helpers of the pass kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>

#include "kernels.h"
#include "passes.cuh"

namespace kg {

// Programmatic dependent launch: pdl_enter waits until the previous kernel of the stream has
// completed and its writes are visible; pdl_leave lets the next kernel's CTAs be scheduled.  The next
// grid launches only after every CTA of this one has passed pdl_leave, so its waiting CTAs never
// hold resources that CTAs of this grid still need.  A kernel launched without the attribute passes
// through both at once.
__device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_leave() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The walk of a pass kernel over its work list.  What does not depend on the previous kernel is done
// before pdl_enter: the first item's descriptor.  The lists and descriptors are written by copies,
// which no kernel launched with the attribute overtakes; after a kernel that writes a descriptor the
// pass is launched without it (LaunchSet::overlap).
template <class Item>
__device__ __forceinline__ void walk_items(const TestDesc *tests, const WorkItem *work, int nwork, int step,
                                           TestDesc *s_desc, ItemCtl *s_ctl, Item &&item) {
    const int first = blockIdx.x;
    if (first < nwork) stage_desc(tests, work[first].test, s_desc, s_ctl);
    pdl_enter();
    for (int wi = first; wi < nwork; wi += gridDim.x) {
        const WorkItem it = work[wi];
        if (wi != first) stage_desc(tests, it.test, s_desc, s_ctl);
        if (step < s_desc->count)
            item(*s_desc, it.unit);  // ends with a barrier
        else
            __syncthreads();  // every thread has read the descriptor
    }
    pdl_leave();
}

inline int set_smem(const void *fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess
               ? 0
               : -1;
}

// The instance for column groups of 2, 4 or 8
template <class K>
K by_group(int G, K g2, K g4, K g8) {
    return G == 2 ? g2 : G == 4 ? g4 : g8;
}

// Pass kernels launch with programmatic stream serialization (each enters through pdl_enter),
// so in a stream or graph the next pass's CTAs are scheduled while the previous pass drains.
// KITE_GB300_PDL=0 launches them plainly.
inline bool pdl_enabled() {
    static const bool on = [] {
        const char *t = getenv("KITE_GB300_PDL");
        return !t || atoi(t) != 0;
    }();
    return on;
}

template <typename... Params, typename... Args>
void launch_pass(const LaunchSet &s, void (*k)(Params...), int grid, size_t smem, Args... args) {
    if (!s.overlap || !pdl_enabled()) {
        k<<<grid, s.threads, smem, s.stream>>>(args...);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(s.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, static_cast<Params>(args)...);
}

}  // namespace kg
