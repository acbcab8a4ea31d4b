// The row pass kernel: rows_item (passes.cuh) over a list of work items, so one launch serves one
// test or a whole batch of tests with different lengths.
#include <cuda_runtime.h>

#include "kernels.h"
#include "launch.cuh"

namespace kg {

template <bool MUL>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_rows(const TestDesc *__restrict__ tests,
                                                   const WorkItem *__restrict__ work, int nwork,
                                                   const int *nwork_dev, int step, double2 *xo,
                                                   const double2 *yo) {
    extern __shared__ longlong2 sm[];
    __shared__ TestDesc s_desc;
    __shared__ ItemCtl s_ctl;
    if (nwork_dev) nwork = *nwork_dev;
    walk_items(tests, work, nwork, step, &s_desc, &s_ctl, [&](const TestDesc &T, int unit) {
        rows_item<MUL, GlobalTables>(T, unit, xo ? xo : T.x, MUL ? (yo ? yo : T.y) : nullptr, sm, s_ctl);
    });
}

void launch_rows(const LaunchSet &s, bool mul, double2 *x, const double2 *y, int step) {
    const size_t smem = s.row_smem_per_lane * (mul ? 6 : 4);
    if (mul)
        launch_pass(s, k_rows<true>, s.grid_rows, smem, s.tests, s.rows, s.nrows, s.nrows_dev, step, x, y);
    else
        launch_pass(s, k_rows<false>, s.grid_rows, smem, s.tests, s.rows, s.nrows, s.nrows_dev, step, x, y);
}

int rows_set_smem(size_t bytes) {
    return set_smem((const void *)k_rows<false>, bytes) | set_smem((const void *)k_rows<true>, bytes);
}

}  // namespace kg
