// The squaring chain of one test run alone (chain.cuh): its launches, and the kernels of a test whose
// items are more than a cluster's.
#include "chain.cuh"

namespace kg {

int chain_set_smem(size_t bytes) {
    int rc = 0;
    for (int G : {2, 4, 8}) {
        const ChainKernel c = chain_cluster_kernel(G);
        rc |= set_smem((const void *)by_group(G, k_chain<1, false>, k_chain<2, false>, k_chain<3, false>), bytes);
        rc |= set_smem((const void *)c, bytes);
        rc |= cudaFuncSetAttribute((const void *)c, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess ? 0 : -1;
    }
    return rc;
}

// The work buffers (a row pair squared takes 4 of the 6 rows of a product), and the tables when they
// are kept: one item of each pass per CTA, one CTA per SM.
static size_t work_smem(const LaunchSet &s) { return std::max(s.row_smem_per_lane * 4, s.col_smem); }
static bool keeps_tables(const LaunchSet &s, int nsm) {
    return std::max(s.nrows, s.ncols) <= nsm && work_smem(s) + s.table_smem <= kMaxChainSmem;
}
size_t chain_smem(const LaunchSet &s, int nsm) { return work_smem(s) + (keeps_tables(s, nsm) ? s.table_smem : 0); }

static int cluster_size(const LaunchSet &s) {
    int size = 1;
    while (size < std::max(s.nrows, s.ncols)) size *= 2;
    return size;
}

static cudaLaunchConfig_t chain_config(const LaunchSet &s, int nsm, int grid, bool cluster, cudaLaunchAttribute *at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = chain_smem(s, nsm);
    cfg.stream = s.stream;
    if (cluster) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = grid;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
    } else {
        at->id = cudaLaunchAttributeCooperative;
        at->val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

bool chain_in_cluster(const LaunchSet &s, int nsm) {
    if (std::max(s.nrows, s.ncols) > kClusterItems) return false;
    // a part of a GPU may have no place for that many CTAs side by side: then cooperatively
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = chain_config(s, nsm, cluster_size(s), true, &at);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, chain_cluster_kernel(s.G), &cfg) == cudaSuccess && clusters > 0) return true;
    (void)cudaGetLastError();
    return false;
}

int chain_grid(const LaunchSet &s, int nsm, bool cluster) {
    if (cluster) return cluster_size(s);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, by_group(s.G, k_chain<1, false>, k_chain<2, false>, k_chain<3, false>),
                                                      kThreads, chain_smem(s, nsm)) != cudaSuccess)
        return 0;
    // as many as there are items, or the fewest that take them in the same number of rounds: the
    // places that are left serve other contexts' kernels
    const int most = std::min(per_sm * nsm, std::max(s.nrows, s.ncols));
    if (most < 1) return 0;
    const auto fewest = [&](int items) {
        const int rounds = (items + most - 1) / most;
        return (items + rounds - 1) / rounds;
    };
    return std::max(fewest(s.nrows), fewest(s.ncols));
}

cudaError_t launch_chain(const LaunchSet &s, int nsm, int grid, bool cluster, double2 *x, int step0, int nsteps, ChainCtl *ctl,
                         unsigned arrived, unsigned *flags, unsigned done, long long limit) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = chain_config(s, nsm, grid, cluster, &at);
    const ChainKernel k = cluster ? chain_cluster_kernel(s.G) : by_group(s.G, k_chain<1, false>, k_chain<2, false>, k_chain<3, false>);
    return cudaLaunchKernelEx(&cfg, k, s.tests, x, step0, nsteps,
                              keeps_tables(s, nsm) ? (int)(work_smem(s) / sizeof(longlong2)) : 0, ctl, arrived, flags, done, limit);
}

}  // namespace kg
