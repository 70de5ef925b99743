/* bulk table kernels for the LayoutK32V64 slot layout (see wc_kernels.cuh) */
#include "wc_tables_pick.cuh"

namespace warpcore {
namespace b200 {

TableKernel table_kernel_k32v64(int W, int op, int fp) { return pick_table_kernel_for<LayoutK32V64>(W, op, fp); }
TableKernel lane_kernel_k32v64(int W, int op) { return pick_lane_kernel_for<LayoutK32V64>(W, op); }
CountInsertKernel count_insert_k32v64(int W) { return pick_count_insert<LayoutK32V64>(W); }

} // namespace b200
} // namespace warpcore
