/*
 * Ray-cast launches of the voxel types other than uint8 and uint16 (int8,
 * int16, uint32, int32, float): one CTA per tile, one kernel per voxel type,
 * filter, edge clamping and look-ahead or lanes per ray (raycast.cu
 * dispatches here).
 */
#include "raycast_device.cuh"

namespace lv
{
namespace
{
template <int DT, int F, int EDGE>
lv_status tiles_launch(lv_ctx* ctx, const RayView& V, const lv_render_launch& L, uint32_t lanes,
                       const uint32_t* order, cudaStream_t s)
{
    if (lanes > 1)
        return split_launch<DT, F, EDGE>(ctx, V, L, lanes, order, s);
    const uint32_t tiles = ((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
    auto k = L.lookahead ? raycast_tiles_kernel<DT, F, EDGE, 1> : raycast_tiles_kernel<DT, F, EDGE, 0>;
    k<<<tiles, L.tile_w * L.tile_h, 0, s>>>(V, L.tile_w, L.tile_h, order);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

template <int DT>
lv_status type_launch(lv_ctx* ctx, const RayView& V, const lv_render_launch& L, uint32_t lanes,
                      const uint32_t* order, cudaStream_t s)
{
    if (V.filter == LV_FILTER_TRILINEAR)
        return V.edge ? tiles_launch<DT, LV_FILTER_TRILINEAR, 1>(ctx, V, L, lanes, order, s)
                      : tiles_launch<DT, LV_FILTER_TRILINEAR, 0>(ctx, V, L, lanes, order, s);
    return V.edge ? tiles_launch<DT, LV_FILTER_NEAREST, 1>(ctx, V, L, lanes, order, s)
                  : tiles_launch<DT, LV_FILTER_NEAREST, 0>(ctx, V, L, lanes, order, s);
}
} // namespace

lv_status launch_other_type(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                            uint32_t lanes, const uint32_t* order, cudaStream_t s)
{
    switch (V.dtype)
    {
    case LV_DT_INT8: return type_launch<LV_DT_INT8>(ctx, V, L, lanes, order, s);
    case LV_DT_INT16: return type_launch<LV_DT_INT16>(ctx, V, L, lanes, order, s);
    case LV_DT_UINT32: return type_launch<LV_DT_UINT32>(ctx, V, L, lanes, order, s);
    case LV_DT_INT32: return type_launch<LV_DT_INT32>(ctx, V, L, lanes, order, s);
    case LV_DT_FLOAT: return type_launch<LV_DT_FLOAT>(ctx, V, L, lanes, order, s);
    default: return fail(ctx, LV_EINVAL, "unknown voxel type");
    }
}

} // namespace lv
