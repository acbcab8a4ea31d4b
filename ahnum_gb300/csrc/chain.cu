// The squaring chain of one test run alone: many squarings in one cooperative launch.
//
// One test's pass is a few dozen to a few hundred work items, each a microsecond or two of work, so
// as launches a squaring is mostly latency: three kernel starts, the descriptor and the tables read
// from L2 again in each.  Here every CTA stays and takes the same items in every squaring, and the
// CTAs meet at a grid-wide barrier after each pass.  When no CTA has more than one item of a pass, it
// keeps the descriptor and its own slices of the tables in shared memory: the barrier's acquire drops
// what L1 held, and a stage that reads its twiddles from L2 takes twice as long.
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

// Copies `count` 16-byte words.
__device__ __forceinline__ void keep(void *dst, const void *src, int count) {
    for (int i = threadIdx.x; i < count; i += blockDim.x) static_cast<int4 *>(dst)[i] = __ldg(static_cast<const int4 *>(src) + i);
}

// The slices of the tables that row pair `unit` and column group `unit` read, from sm[at] on, and the
// descriptor's pointers to them (such that the passes find them under their own indices).
template <int LG>
__device__ __forceinline__ void keep_tables(TestDesc *d, longlong2 *buf, int unit, int at) {
    const int R = d->R, C = d->C, G = 1 << LG, points = R << LG;
    int4 *twr = reinterpret_cast<int4 *>(buf + at), *twc = twr + C, *sw = twc + R, *t4 = sw + C;
    int4 *osc = t4 + points, *w = osc + points, *bits = w + points;
    keep(twr, d->twr, C - 1);
    keep(twc, d->twc, R - 1);
    const int row = unit < d->npairs ? d->pairs[unit].x : 0;
    if (unit < d->npairs) keep(sw, d->sw + (size_t)row * C, C);
    if (unit < d->NG) {
        for (int i = threadIdx.x; i < points; i += blockDim.x) {
            const size_t e = (size_t)(i >> LG) * C + (unit << LG) + (i & (G - 1));
            t4[i] = __ldg(d->t4 + e);
            osc[i] = __ldg(reinterpret_cast<const int4 *>(d->osc) + e);
            w[i] = __ldg(reinterpret_cast<const int4 *>(d->w) + e);
            reinterpret_cast<unsigned short *>(bits)[i] = __ldg(reinterpret_cast<const unsigned short *>(d->bits) + e);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const ptrdiff_t first = (ptrdiff_t)unit << LG;  // the group's first column
        d->twr = twr;
        d->twc = twc;
        d->sw = sw - (ptrdiff_t)row * C;
        d->pitch = G;
        d->t4 = t4 - first;
        d->osc = reinterpret_cast<long long *>(osc - first);
        d->w = reinterpret_cast<long long *>(w - first);
        d->bits = reinterpret_cast<uint8_t *>(bits) - 2 * first;
    }
    __syncthreads();
}

template <int LG>
__global__ void __launch_bounds__(kThreads, 2) k_chain(const TestDesc *__restrict__ test, double2 *x, int step0, int nsteps,
                                                       int tables_at, ChainCtl *ctl, unsigned arrived, long long limit) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    const TestDesc &T = stage_desc(test, 0, &s_desc, &s_ctl);
    const int np = T.npairs, ng = T.NG;
    if (tables_at) keep_tables<LG>(&s_desc, sm, blockIdx.x, tables_at);
    for (int s = 0; s < nsteps; s++) {
        for (int u = blockIdx.x; u < np; u += gridDim.x) {
            clear_ctl(&s_ctl);
            rows_item<false, AnyTables>(T, u, x, nullptr, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            clear_ctl(&s_ctl);
            col_inverse_item<LG, AnyTables>(T, g, step0 + s, x, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            clear_ctl(&s_ctl);
            col_forward_item<LG, AnyTables>(T, g, x, true, T.digit_bits, sm, s_ctl);
        }
        if (!grid_barrier(ctl, arrived += gridDim.x, limit)) return;
    }
}

int chain_set_smem(size_t bytes) {
    return set_smem((const void *)k_chain<1>, bytes) | set_smem((const void *)k_chain<2>, bytes) |
           set_smem((const void *)k_chain<3>, bytes);
}

// The work buffers (a row pair squared takes 4 of the 6 rows of a product), and the tables when they
// are kept: one item of each pass per CTA, one CTA per SM.
static size_t work_smem(const LaunchSet &s) { return std::max(s.row_smem_per_lane * 4, s.col_smem); }
static bool keeps_tables(const LaunchSet &s, int nsm) {
    return std::max(s.nrows, s.ncols) <= nsm && work_smem(s) + s.table_smem <= kMaxChainSmem;
}
size_t chain_smem(const LaunchSet &s, int nsm) { return work_smem(s) + (keeps_tables(s, nsm) ? s.table_smem : 0); }

int chain_grid(const LaunchSet &s, int nsm) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, by_group(s.G, k_chain<1>, k_chain<2>, k_chain<3>), kThreads,
                                                      chain_smem(s, nsm)) != cudaSuccess)
        return 0;
    return std::min(per_sm * nsm, std::max(s.nrows, s.ncols));
}

cudaError_t launch_chain(const LaunchSet &s, int nsm, int grid, double2 *x, int step0, int nsteps, ChainCtl *ctl, unsigned arrived,
                         long long limit) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = chain_smem(s, nsm);
    cfg.stream = s.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, by_group(s.G, k_chain<1>, k_chain<2>, k_chain<3>), s.tests, x, step0, nsteps,
                              keeps_tables(s, nsm) ? (int)(work_smem(s) / sizeof(longlong2)) : 0, ctl, arrived, limit);
}

}  // namespace kg
