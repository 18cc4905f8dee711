/*
 * Ray-cast kernels of the voxel types other than uint8 and uint16 (int8,
 * int16, uint32, int32, float): one CTA per tile, one kernel per voxel type,
 * filter, edge clamping and look-ahead or lanes per ray (raycast.cu launches
 * them).
 */
#include "raycast_device.cuh"

namespace lv
{
namespace
{
template <int DT, int F, int EDGE>
TileKernel edge_kernel(const RayLaunch& R)
{
    if (R.lanes > 1)
        return split_kernel_of<DT, F, EDGE>(R.lanes);
    return R.shape.lookahead ? raycast_tiles_kernel<DT, F, EDGE, 1>
                             : raycast_tiles_kernel<DT, F, EDGE, 0>;
}

template <int DT>
TileKernel type_kernel(const RayView& V, const RayLaunch& R)
{
    if (V.filter == LV_FILTER_TRILINEAR)
        return V.edge ? edge_kernel<DT, LV_FILTER_TRILINEAR, 1>(R)
                      : edge_kernel<DT, LV_FILTER_TRILINEAR, 0>(R);
    return V.edge ? edge_kernel<DT, LV_FILTER_NEAREST, 1>(R)
                  : edge_kernel<DT, LV_FILTER_NEAREST, 0>(R);
}
} // namespace

TileKernel other_type_kernel(const RayView& V, const RayLaunch& R)
{
    switch (V.dtype)
    {
    case LV_DT_INT8: return type_kernel<LV_DT_INT8>(V, R);
    case LV_DT_INT16: return type_kernel<LV_DT_INT16>(V, R);
    case LV_DT_UINT32: return type_kernel<LV_DT_UINT32>(V, R);
    case LV_DT_INT32: return type_kernel<LV_DT_INT32>(V, R);
    case LV_DT_FLOAT: return type_kernel<LV_DT_FLOAT>(V, R);
    default: return nullptr;
    }
}

} // namespace lv
