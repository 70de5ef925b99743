/* bulk table kernels for the LayoutSet64 slot layout (see wc_kernels.cuh) */
#include "wc_tables_pick.cuh"

namespace warpcore {
namespace b200 {

TableKernel table_kernel_set64(int W, int op, int fp) { return pick_table_kernel_for<LayoutSet64>(W, op, fp); }
TableKernel lane_kernel_set64(int W, int op) { return pick_lane_kernel_for<LayoutSet64>(W, op); }

} // namespace b200
} // namespace warpcore
