/*
 * Ray-cast launches of uint8 and uint16 volumes with several lanes per ray
 * (raycast_split_kernel), one kernel per voxel type, filter, edge clamping or
 * fixed pitch, and lanes (raycast.cu dispatches here).
 */
#include "raycast_device.cuh"

namespace lv
{
namespace
{
template <int DT>
lv_status type_split(lv_ctx* ctx, const RayView& V, const lv_render_launch& L, uint32_t lanes,
                     uint32_t pitch, const uint32_t* order, cudaStream_t s)
{
    if (V.filter != LV_FILTER_TRILINEAR)
        return V.edge ? split_launch<DT, LV_FILTER_NEAREST, 1>(ctx, V, L, lanes, order, s)
                      : split_launch<DT, LV_FILTER_NEAREST, 0>(ctx, V, L, lanes, order, s);
    switch (pitch)
    {
    case 34: return split_launch<DT, LV_FILTER_TRILINEAR, 34>(ctx, V, L, lanes, order, s);
    case 66: return split_launch<DT, LV_FILTER_TRILINEAR, 66>(ctx, V, L, lanes, order, s);
    case 130: return split_launch<DT, LV_FILTER_TRILINEAR, 130>(ctx, V, L, lanes, order, s);
    default:
        return V.edge ? split_launch<DT, LV_FILTER_TRILINEAR, 1>(ctx, V, L, lanes, order, s)
                      : split_launch<DT, LV_FILTER_TRILINEAR, 0>(ctx, V, L, lanes, order, s);
    }
}
} // namespace

lv_status launch_split(lv_ctx* ctx, const RayView& V, const lv_render_launch& L, uint32_t lanes,
                       uint32_t pitch, const uint32_t* order, cudaStream_t s)
{
    return V.dtype == LV_DT_UINT8 ? type_split<LV_DT_UINT8>(ctx, V, L, lanes, pitch, order, s)
                                  : type_split<LV_DT_UINT16>(ctx, V, L, lanes, pitch, order, s);
}

} // namespace lv
