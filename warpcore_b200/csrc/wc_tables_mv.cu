/* MultiValueHashTable kernels for the u32/u32 and u64/u64 layouts (see wc_mv.cuh) */
#include "wc_mv_pick.cuh"

namespace warpcore {
namespace b200 {

MvKernels mv_kernels(int layout, int W)
{
    if (layout == kLayoutKV32) return mv_pick_w<LayoutKV32>(W);
    if (layout == kLayoutKV64) return mv_pick_w<LayoutKV64>(W);
    if (layout == kLayoutK32V64 || layout == kLayoutK64V32) return mv_kernels_mixed(layout, W);
    return MvKernels{};
}

const void *multi_dry_status_kernel_ptr()
{
    return reinterpret_cast<const void *>(multi_dry_status_kernel<0>);
}

} // namespace b200
} // namespace warpcore
