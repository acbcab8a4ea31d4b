// The squaring chain of a short test in one thread-block cluster (chain.cuh).
#include "chain.cuh"

namespace kg {

ChainKernel chain_cluster_kernel(int G) { return by_group(G, k_chain<1, true>, k_chain<2, true>, k_chain<3, true>); }

}  // namespace kg
