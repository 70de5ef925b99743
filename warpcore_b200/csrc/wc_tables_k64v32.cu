/* bulk table kernels for the LayoutK64V32 slot layout (see wc_kernels.cuh) */
#include "wc_tables_pick.cuh"

namespace warpcore {
namespace b200 {

TableKernel table_kernel_k64v32(int W, int op, int fp) { return pick_table_kernel_for<LayoutK64V32>(W, op, fp); }
TableKernel lane_kernel_k64v32(int W, int op) { return pick_lane_kernel_for<LayoutK64V32>(W, op); }
CountInsertKernel count_insert_k64v32(int W) { return pick_count_insert<LayoutK64V32>(W); }

} // namespace b200
} // namespace warpcore
