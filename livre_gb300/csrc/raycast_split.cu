/*
 * Ray-cast kernels of uint8 and uint16 volumes with several lanes per ray
 * (raycast_split_kernel), one per voxel type, filter, edge clamping or fixed
 * pitch, and lanes (raycast.cu launches them).
 */
#include "raycast_device.cuh"

namespace lv
{
namespace
{
template <int DT>
TileKernel type_kernel(const RayView& V, uint32_t lanes, uint32_t pitch)
{
    if (V.filter != LV_FILTER_TRILINEAR)
        return V.edge ? split_kernel_of<DT, LV_FILTER_NEAREST, 1>(lanes)
                      : split_kernel_of<DT, LV_FILTER_NEAREST, 0>(lanes);
    switch (pitch)
    {
    case 34: return split_kernel_of<DT, LV_FILTER_TRILINEAR, 34>(lanes);
    case 66: return split_kernel_of<DT, LV_FILTER_TRILINEAR, 66>(lanes);
    case 130: return split_kernel_of<DT, LV_FILTER_TRILINEAR, 130>(lanes);
    default:
        return V.edge ? split_kernel_of<DT, LV_FILTER_TRILINEAR, 1>(lanes)
                      : split_kernel_of<DT, LV_FILTER_TRILINEAR, 0>(lanes);
    }
}
} // namespace

TileKernel split_kernel(const RayView& V, uint32_t lanes, uint32_t pitch)
{
    return V.dtype == LV_DT_UINT8 ? type_kernel<LV_DT_UINT8>(V, lanes, pitch)
                                  : type_kernel<LV_DT_UINT16>(V, lanes, pitch);
}

} // namespace lv
