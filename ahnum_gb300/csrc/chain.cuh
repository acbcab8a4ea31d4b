// The squaring chain of one test run alone: many squarings in one launch.
//
// One test's pass is a few dozen to a few hundred work items, each a microsecond or two of work, so
// as launches a squaring is mostly latency: three kernel starts, the descriptor and the tables read
// from L2 again in each.  Here every CTA stays and takes the same items in every squaring.  When no CTA
// has more than one item of a pass, it keeps the descriptor, its own slices of the tables and its digits
// in shared memory: a barrier's acquire drops what L1 held, and a stage that reads its twiddles from L2
// takes twice as long.
//
// A row pass needs every column group and a column pass every row pair, so all CTAs meet after each of
// them.  Between the two halves of the column pass a group only needs its left neighbour's carries (the
// first one the last one's, and the fold): it waits for that group's flag.
//
// Two kinds of meeting (CLUSTER).  Up to kClusterItems items: the CTAs are one thread-block cluster and
// meet at its hardware barrier.  More: a cooperative launch, and a counter in global memory.
// us per squaring on GB300, best shape, with three grid barriers -> neighbour's flag -> cluster:
// 512 digits 11.7 -> 11.7 -> 9.6, 896 digits 13.4 -> 12.9 -> 11.3, 1344 digits 14.0 -> 12.8 -> 12.3,
// 27648 digits 15.6 -> 15.3, 49152 digits 15.9 -> 15.2, 1769472 digits 111 -> 109.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "passes.cuh"

namespace kg {

// Thread 0 polls `word` until it has reached `need` (modulo 2^32); what was written before a release of
// that value is visible after, to the CTA.  Every CTA is resident (cooperative launch), so the wait
// ends; if it does not within `limit` SM cycles, or another CTA has given up, the chain ends and says so.
__device__ __forceinline__ bool wait_for(const unsigned *word, unsigned need, ChainCtl *ctl, long long limit) {
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned v;
        const long long t0 = clock64();
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
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

// All CTAs of the grid have arrived `need` times at ctl->arrived, or at the cluster's barrier once more.
template <bool CLUSTER>
__device__ __forceinline__ bool meet(ChainCtl *ctl, unsigned need, long long limit) {
    if constexpr (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    } else {
        __syncthreads();
        if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->arrived) : "memory");
        return wait_for(&ctl->arrived, need, ctl, limit);
    }
}

// Copies `count` 16-byte words.
__device__ __forceinline__ void keep(void *dst, const void *src, int count) {
    for (int i = threadIdx.x; i < count; i += blockDim.x) static_cast<int4 *>(dst)[i] = __ldg(static_cast<const int4 *>(src) + i);
}

// The slices of the tables that row pair `unit` and column group `unit` read, from sm[at] on, room for
// the group's digits, and the descriptor's pointers to them (such that the passes find them under their
// own indices).
template <int LG>
__device__ __forceinline__ void keep_tables(TestDesc *d, longlong2 *buf, int unit, int at) {
    const int R = d->R, C = d->C, G = 1 << LG, points = R << LG;
    const ptrdiff_t first = (ptrdiff_t)unit << LG;  // the group's first column
    int4 *twr = reinterpret_cast<int4 *>(buf + at), *twc = twr + C, *sw = twc + R, *t4 = sw + C;
    int4 *osc = t4 + points, *w = osc + points, *dig = w + points, *bits = dig + points;
    keep(twr, d->twr, C - 1);
    keep(twc, d->twc, R - 1);
    const int row = unit < d->npairs ? d->pairs[unit].x : 0;
    if (unit < d->npairs) keep(sw, d->sw + (size_t)row * C, C);
    if (unit < d->NG) {
        for (int i = threadIdx.x; i < points; i += blockDim.x) {
            const size_t e = (size_t)(i >> LG) * C + (unit << LG) + (i & (G - 1));
            t4[i] = __ldg(d->t4 + e);
            osc[i] = __ldg(reinterpret_cast<const int4 *>(d->osc) + e);
        }
        keep(w, reinterpret_cast<const int4 *>(d->w) + first * R, points);
        const unsigned *widths = reinterpret_cast<const unsigned *>(d->segbits + 2 * first * R);
        for (int i = threadIdx.x; i < points / 2; i += blockDim.x) reinterpret_cast<unsigned *>(bits)[i] = __ldg(widths + i);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        d->twr = twr;
        d->twc = twc;
        d->sw = sw - (ptrdiff_t)row * C;
        d->pitch = G;
        d->t4 = t4 - first;
        d->osc = reinterpret_cast<long long *>(osc - first);
        d->w = reinterpret_cast<long long *>(w - first * R);
        d->segbits = reinterpret_cast<uint8_t *>(bits) - 2 * first * R;
        d->dig = reinterpret_cast<long long *>(dig - first * R);
    }
    __syncthreads();
}

// arrived: of ctl->arrived before the launch; flags: of each column group, kFlagWords apart, all equal to
// `done`, the squarings of chains so far.
template <int LG, bool CLUSTER>
__global__ void __launch_bounds__(kThreads, 2) k_chain(const TestDesc *__restrict__ test, double2 *x, int step0, int nsteps,
                                                       int tables_at, ChainCtl *ctl, unsigned arrived, unsigned *flags,
                                                       unsigned done, long long limit) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    const TestDesc &T = stage_desc(test, 0, &s_desc, &s_ctl);
    const int np = T.npairs, ng = T.NG;
    // The row exponents' largest alternates between two words: the one that the next squaring will use
    // is cleared in the second half of the column pass, when every CTA has read it.
    int *const emax = T.emax;
    if (tables_at) keep_tables<LG>(&s_desc, sm, blockIdx.x, tables_at);
    for (int s = 0; s < nsteps; s++) {
        for (int u = blockIdx.x; u < np; u += gridDim.x) {
            clear_ctl(&s_ctl);
            rows_item<false, AnyTables>(T, u, x, nullptr, sm, s_ctl);
        }
        if (!meet<CLUSTER>(ctl, arrived += gridDim.x, limit)) return;
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            clear_ctl(&s_ctl);
            col_inverse_item<LG, AnyTables>(T, g, step0 + s, x, sm, s_ctl);  // ends with a barrier
            if (!CLUSTER && threadIdx.x == 0)
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flags + g * kFlagWords), "r"(done + s + 1) : "memory");
        }
        if (CLUSTER) meet<true>(ctl, 0, 0);
        if (threadIdx.x == 0) s_desc.emax = emax + ((s + 1) & 1);
        for (int g = blockIdx.x; g < ng; g += gridDim.x) {
            if (!CLUSTER && !wait_for(flags + (g ? g - 1 : ng - 1) * kFlagWords, done + s + 1, ctl, limit)) return;
            clear_ctl(&s_ctl);
            col_forward_item<LG, AnyTables>(T, g, x, true, T.digit_bits, sm, s_ctl);
        }
        if (!meet<CLUSTER>(ctl, arrived += gridDim.x, limit)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // both words clear between chains
        emax[0] = INT_MIN;
        emax[1] = INT_MIN;
    }
}

using ChainKernel = void (*)(const TestDesc *, double2 *, int, int, int, ChainCtl *, unsigned, unsigned *, unsigned, long long);
ChainKernel chain_cluster_kernel(int G);  // chain_cluster.cu

}  // namespace kg
