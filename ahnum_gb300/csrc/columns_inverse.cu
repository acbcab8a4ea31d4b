// The kernels of the column inverse: the first half of the column pass, and the digits of a number.
// Each walks a list of work items, as the row pass does.
#include <cuda_runtime.h>

#include "kernels.h"
#include "launch.cuh"

namespace kg {

template <int LG>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_col_inverse(const TestDesc *__restrict__ tests,
                                                          const WorkItem *__restrict__ work,
                                                          int nwork, const int *nwork_dev,
                                                          int step, const double2 *xo) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    if (nwork_dev) nwork = *nwork_dev;
    walk_items(
        tests, work, nwork, step, &s_desc, &s_ctl,
        [&](const TestDesc &T, int g) { col_inverse_item<LG, GlobalTables>(T, g, step, xo ? xo : T.x, sm, s_ctl); });
}

template <int LG>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_col_digits(const TestDesc *__restrict__ tests,
                                                         const WorkItem *__restrict__ work,
                                                         int nwork, const double2 *xo, long long *digo) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    walk_items(
        tests, work, nwork, 0, &s_desc, &s_ctl,
        [&](const TestDesc &T, int g) { col_digits_item<LG, GlobalTables>(T, g, xo ? xo : T.x, digo ? digo : T.dig, sm, s_ctl); });
}

void launch_col_inverse(const LaunchSet &s, const double2 *x, int step) {
    launch_pass(s, by_group(s.G, k_col_inverse<1>, k_col_inverse<2>, k_col_inverse<3>), s.grid_cols, s.col_smem, s.tests, s.cols, s.ncols,
                s.ncols_dev, step, x);
    if (s.narrow)
        launch_pass(s, k_col_inverse<2>, s.grid_cols, s.col_smem, s.tests, s.cols4, 0, s.ncols4_dev, step, x);
}

void launch_col_digits(const LaunchSet &s, const double2 *x, long long *dig) {
    launch_pass(s, by_group(s.G, k_col_digits<1>, k_col_digits<2>, k_col_digits<3>), s.grid_cols, s.col_smem, s.tests, s.cols, s.ncols, x, dig);
}

int col_inverse_set_smem(size_t bytes) {
    return set_smem((const void *)k_col_inverse<1>, bytes) | set_smem((const void *)k_col_inverse<2>, bytes) |
           set_smem((const void *)k_col_inverse<3>, bytes) | set_smem((const void *)k_col_digits<1>, bytes) | set_smem((const void *)k_col_digits<2>, bytes) |
           set_smem((const void *)k_col_digits<3>, bytes);
}

}  // namespace kg
