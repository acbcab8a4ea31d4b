// The kernel of the column forward: the second half of the column pass, over a list of work items.
#include <cuda_runtime.h>

#include "kernels.h"
#include "launch.cuh"

namespace kg {

template <int LG>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_col_forward(const TestDesc *__restrict__ tests,
                                                          const WorkItem *__restrict__ work,
                                                          int nwork, const int *nwork_dev, int step,
                                                          double2 *xo, int use_slots, int digit_bits) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    if (nwork_dev) nwork = *nwork_dev;
    walk_items(
        tests, work, nwork, step, &s_desc, &s_ctl,
        [&](const TestDesc &T, int g) {
            col_forward_item<LG, GlobalTables>(T, g, xo ? xo : T.x, use_slots != 0, digit_bits > 0 ? digit_bits : T.digit_bits, sm, s_ctl);
        });
}

void launch_col_forward(const LaunchSet &s, double2 *x, bool use_slots, int step, int digit_bits) {
    launch_pass(s, by_group(s.G, k_col_forward<1>, k_col_forward<2>, k_col_forward<3>), s.grid_cols, s.col_smem, s.tests, s.cols, s.ncols,
                s.ncols_dev, step, x, use_slots ? 1 : 0, digit_bits);
    if (s.narrow)
        launch_pass(s, k_col_forward<2>, s.grid_cols, s.col_smem, s.tests, s.cols4, 0, s.ncols4_dev, step, x, use_slots ? 1 : 0, digit_bits);
}

int col_forward_set_smem(size_t bytes) { return set_smem((const void *)k_col_forward<1>, bytes) | set_smem((const void *)k_col_forward<2>, bytes) |
           set_smem((const void *)k_col_forward<3>, bytes); }

}  // namespace kg
