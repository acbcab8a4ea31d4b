// The persistent squaring kernel: many squarings of every test of the work lists in one launch
// (see passes.cuh for the passes it runs).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "passes.cuh"

namespace kg {

// Waits until *ctr >= need, reading it with acquire semantics at GPU scope.  Gives up (returns
// false) when another CTA has raised *flag, or after `limit` SM cycles, raising *flag itself.
__device__ __noinline__ bool wait_count(const unsigned *ctr, unsigned need, unsigned *flag, long long limit) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
    if (v >= need) return true;
    const long long t0 = clock64();
    for (;;) {
        __nanosleep(128);
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= need) return true;
        if (*(volatile const unsigned *)flag) return false;
        if (clock64() - t0 > limit) {
            atomicOr(flag, 1u);
            return false;
        }
    }
}

// `nsteps` squarings of every test of the work lists in one persistent launch.
//
// The work is one queue, taken in order by atomically incrementing flow[kFlowNext]: for each
// step, every row pair, then every column group (inverse half), then every column group
// (forward half).  A CTA that takes an item first waits until the test's previous phase is
// complete: flow[kFlowDone + test] counts the test's finished items, and the phases of one test
// follow each other, so item counts alone say which phase is done.  Different tests overlap
// freely, so no CTA idles at the end of a phase or of a step, as it would at the end of a
// kernel launch.  Every wait is on items earlier in the queue, which CTAs already running hold,
// so each wait ends; one that runs out of time raises flow[kFlowTimeout] and every CTA returns.
// MIXED: after `cols` come the items of tests with groups of 4 columns, `cols4`.
template <int LG, bool MIXED>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_squarings(const TestDesc *__restrict__ tests,
                                                        const WorkItem *__restrict__ rows, int nrows,
                                                        const int *nrows_dev,
                                                        const WorkItem *__restrict__ cols, int ncols,
                                                        const int *ncols_dev, const WorkItem *__restrict__ cols4,
                                                        const int *ncols4_dev, int step0, int nsteps,
                                                        unsigned *flow, long long wait_limit) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    __shared__ unsigned s_q;
    __shared__ int s_ok;
    const unsigned nr = (unsigned)(nrows_dev ? *nrows_dev : nrows);
    const unsigned n8 = (unsigned)(ncols_dev ? *ncols_dev : ncols), nc = n8 + (MIXED ? (unsigned)*ncols4_dev : 0);
    const auto item_at = [&](unsigned r) {
        if (r < nr) return rows[r];
        const unsigned c = (r - nr) % nc;
        return MIXED && c >= n8 ? cols4[c - n8] : cols[c];
    };
    const unsigned per_step = nr + 2 * nc;
    const unsigned total = per_step * (unsigned)nsteps;
    for (;;) {
        __syncthreads();  // every thread has read the previous item's s_q
        if (threadIdx.x == 0) {
            const unsigned q = atomicAdd(&flow[kFlowNext], 1u);
            int ok = 1;
            if (q < total) {
                const unsigned st = q / per_step, r = q % per_step;
                const WorkItem it = item_at(r);
                const TestDesc &T = tests[it.test];
                unsigned need = st * (unsigned)(T.npairs + 2 * T.NG);
                if (r >= nr) need += (unsigned)T.npairs;
                if (r >= nr + nc) need += (unsigned)T.NG;
                ok = wait_count(&flow[kFlowDone + it.test], need, &flow[kFlowTimeout], wait_limit);
            }
            s_q = q;
            s_ok = ok;
        }
        __syncthreads();
        const unsigned q = s_q;
        if (q >= total || !s_ok) return;
        const unsigned st = q / per_step, r = q % per_step;
        const WorkItem it = item_at(r);
        const TestDesc &T = stage_desc(tests, it.test, &s_desc, &s_ctl);
        const int step = step0 + (int)st;
        if (step < T.count) {
            if (r < nr)
                rows_item<false, GlobalTables>(T, it.unit, T.x, nullptr, sm, s_ctl);
            else if (MIXED && T.G == 4 && r < nr + nc)
                col_inverse_item<2, GlobalTables>(T, it.unit, step, T.x, sm, s_ctl);
            else if (MIXED && T.G == 4)
                col_forward_item<2, GlobalTables>(T, it.unit, T.x, true, T.digit_bits, sm, s_ctl);
            else if (r < nr + nc)
                col_inverse_item<LG, GlobalTables>(T, it.unit, step, T.x, sm, s_ctl);
            else
                col_forward_item<LG, GlobalTables>(T, it.unit, T.x, true, T.digit_bits, sm, s_ctl);
        }
        // each item ends with a barrier after its last global write (but for thread 0's own):
        // publish them, then count
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(&flow[kFlowDone + it.test], 1u);
        }
    }
}

// shared memory of k_squarings: a row pair squared (4 lanes of the longest row; row_smem is
// sized for the 6 lanes of a product) or a column group
size_t squarings_smem(size_t row_smem, size_t col_smem) { return std::max(row_smem / 6 * 4, col_smem); }

using SquaringsKernel = void (*)(const TestDesc *, const WorkItem *, int, const int *, const WorkItem *, int, const int *, const WorkItem *,
                                 const int *, int, int, unsigned *, long long);
static SquaringsKernel kernel_of(const LaunchSet &s) {
    return s.narrow ? k_squarings<3, true> : by_group(s.G, k_squarings<1, false>, k_squarings<2, false>, k_squarings<3, false>);
}

int squarings_set_smem(size_t bytes) {
    return set_smem((const void *)k_squarings<1, false>, bytes) | set_smem((const void *)k_squarings<2, false>, bytes) |
           set_smem((const void *)k_squarings<3, false>, bytes) | set_smem((const void *)k_squarings<3, true>, bytes);
}

int squarings_grid(const LaunchSet &s, int nsm) {
    int per_sm = 0;
    const size_t smem = squarings_smem(s.row_smem_per_lane * 6, s.col_smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_of(s), s.threads, smem) != cudaSuccess) return 0;
    return per_sm * nsm;
}

int launch_squarings(const LaunchSet &s, unsigned *flow, int step0, int nsteps, int grid, long long wait_limit) {
    if (grid < 1) return -1;
    const size_t smem = squarings_smem(s.row_smem_per_lane * 6, s.col_smem);
    kernel_of(s)<<<grid, s.threads, smem, s.stream>>>(s.tests, s.rows, s.nrows, s.nrows_dev, s.cols, s.ncols, s.ncols_dev, s.cols4,
                                                      s.ncols4_dev, step0, nsteps, flow, wait_limit);
    return 0;
}

}  // namespace kg
