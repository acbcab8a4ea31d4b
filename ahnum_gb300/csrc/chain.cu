// The squaring chain of one test run alone: many squarings in one cooperative launch.
//
// One test's pass is a few dozen to a few hundred work items, each a microsecond or two of work, so
// as launches a squaring is mostly latency: three kernel starts, the descriptor and the tables read
// from L2 again in each, the instruction cache filled again in each.  Here every CTA stays: it takes
// the same items in every squaring, so that its descriptor stays in shared memory and its slices of
// the tables in L1, and the CTAs meet at a grid-wide barrier after each pass.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "passes.cuh"

namespace kg {

// All CTAs of the grid have arrived `need` times at ctl->arrived (modulo 2^32); what they wrote before
// is visible after.  Every CTA is resident (cooperative launch), so the wait ends; if it does not
// within `limit` SM cycles, or another CTA has given up, the chain ends and says so.
__device__ __forceinline__ bool grid_barrier(ChainCtl *ctl, unsigned need, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned v;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->arrived) : "memory");
        const long long t0 = clock64();
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->arrived) : "memory");
            if ((int)(v - need) >= 0) break;
            if (*(volatile unsigned *)&ctl->timeout || clock64() - t0 > limit) {
                atomicOr(&ctl->timeout, 1u);
                *(volatile unsigned *)ctl->host_timeout = 1u;
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

template <int LG>
__global__ void __launch_bounds__(kThreads, 2) k_chain(const TestDesc *__restrict__ test, double2 *x, int step0, int nsteps,
                                                       ChainCtl *ctl, unsigned arrived, long long limit) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    const TestDesc &T = stage_desc(test, 0, &s_desc, &s_ctl);
    const int np = T.npairs, ng = T.NG;
    for (int s = 0; s < nsteps; s++) {
        for (int u = blockIdx.x; u < np; u += gridDim.x) {
            clear_ctl(&s_ctl);
            rows_item<false>(T, u, x, nullptr, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            clear_ctl(&s_ctl);
            col_inverse_item<LG>(T, g, step0 + s, x, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            clear_ctl(&s_ctl);
            col_forward_item<LG>(T, g, x, true, T.digit_bits, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
    }
}

int chain_set_smem(size_t bytes) {
    return set_smem((const void *)k_chain<1>, bytes) | set_smem((const void *)k_chain<2>, bytes) |
           set_smem((const void *)k_chain<3>, bytes);
}

// a row pair squared takes 4 of the 6 rows of a product's
static size_t chain_smem(const LaunchSet &s) { return std::max(s.row_smem_per_lane * 4, s.col_smem); }

int chain_grid(const LaunchSet &s, int nsm) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, by_group(s.G, k_chain<1>, k_chain<2>, k_chain<3>), kThreads,
                                                      chain_smem(s)) != cudaSuccess)
        return 0;
    return std::min(per_sm * nsm, std::max(s.nrows, s.ncols));
}

cudaError_t launch_chain(const LaunchSet &s, int grid, double2 *x, int step0, int nsteps, ChainCtl *ctl, unsigned arrived,
                         long long limit) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = chain_smem(s);
    cfg.stream = s.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, by_group(s.G, k_chain<1>, k_chain<2>, k_chain<3>), s.tests, x, step0, nsteps, ctl, arrived,
                              limit);
}

}  // namespace kg
