/*
 * Per-brick value histograms on the device.
 *
 * Restates HistogramObject (livre/lib/cache/HistogramObject.cpp:30-224) and
 * the accumulation of HistogramFilter::execute (livre/lib/pipeline/
 * HistogramFilter.cpp:78-149) for one full viewport:
 *  - only the brick's own voxels count (the overlap is skipped);
 *  - each count is weighted by the number of finest-level voxels one voxel of
 *    the brick stands for, (2^(depth - 1 - level))^3;
 *  - the bin of value v over n bins and the data range [lo, hi] is
 *    floor((v - lo) * (n - 1) / (hi - lo)), clamped to [0, n - 1]; for uint8
 *    with 256 bins over [0, 255] this is the reference's bin = v. (The
 *    reference's integer bin width for 16-bit data divides by zero or writes
 *    past its bins for small or large ranges; the same formula is used for
 *    every type here.)
 * One or more CTAs per brick build its histogram in shared memory from the brick in
 * the HBM pool, then adds it (64-bit) to the per-brick and accumulated
 * outputs.
 */
#include <algorithm>
#include <vector>

#include "lv_runtime.h"

namespace
{
using namespace lv;

struct HistJob
{
    uint64_t offset; /* brick byte offset in the pool */
    uint64_t scale;  /* finest voxels per brick voxel */
};

constexpr uint32_t kHistThreads = 256;
constexpr uint32_t kHistWarps = kHistThreads / 32;
constexpr uint32_t kHistRows = 8; /* rows whose loads a lane has in flight */
/* 32-bit counters of a block in shared memory */
constexpr uint32_t kHistCounters = 8192;
/* blocks launched per SM: two rounds of the 5 resident ones, so that the SMs
 * end together */
constexpr uint32_t kHistBlocksPerSm = 10;
constexpr uint64_t kHistKeep = 64u << 20; /* bytes of counts a context keeps room for */

/* Voxels counted by value first: uint8 and int8, 32 counters per value. */
constexpr uint32_t kValueCopiesLog2 = 5;
constexpr bool by_value(int dt) { return dt == LV_DT_UINT8 || dt == LV_DT_INT8; }

/* The value of `bits` (a voxel, zero-extended) as a float. */
template <int DT>
__device__ __forceinline__ float voxel_value(uint32_t bits)
{
    switch (DT)
    {
    case LV_DT_INT8: return float(int8_t(bits));
    case LV_DT_INT16: return float(int16_t(bits));
    case LV_DT_INT32: return __int2float_rn(int32_t(bits));
    case LV_DT_FLOAT: return __uint_as_float(bits);
    default: return __uint2float_rn(bits);
    }
}

template <int DT>
__device__ __forceinline__ uint32_t load_voxel(const uint8_t* brick, uint32_t idx)
{
    if (DT == LV_DT_UINT8 || DT == LV_DT_INT8)
        return __ldg(brick + idx);
    if (DT == LV_DT_UINT16 || DT == LV_DT_INT16)
        return __ldg(reinterpret_cast<const uint16_t*>(brick) + idx);
    return __ldg(reinterpret_cast<const uint32_t*>(brick) + idx);
}

__device__ __forceinline__ uint32_t bin_of(float v, float lo, float scale_bins, uint32_t n_bins)
{
    const float f = floorf((v - lo) * scale_bins);
    return uint32_t(int(fminf(fmaxf(f, 0.0f), float(n_bins - 1))));
}

/* A brick's voxels without the overlap, N voxels per row and slice stored,
 * overlap O, B counted. */
struct HistBrick
{
    uint32_t N0, N1, O0, O1, O2, B0, B1, B2;
};

/* Histogram of bricks: blockIdx.x is the brick, gridDim.y blocks share its
 * rows. Bound by reading the bricks; what stood in the way was counting:
 * one shared counter per bin, which the many voxels of equal value (a dark
 * ground) serialise on, and an index division per voxel. So
 *  - a bin has `1 << copies_log2` counters and lane l uses copy l: with 32
 *    copies (up to 256 bins) a warp's counts hit 32 banks whatever the data;
 *  - 8-bit voxels count their 256 values, and each value's count goes to its
 *    bin once at the end;
 *  - a warp takes whole rows (several short ones), coordinates advancing
 *    without a division, kHistRows loads in flight;
 *  - QUADS, bricks stored as voxel quads (quad_layout): the element at even
 *    (x, y) holds the four voxels of its 2 x 2 square, so every second row
 *    of elements is read.
 * 512 bricks of 64^3 uint8 voxels in quads: 561 -> 85 us (4 rows in flight: 103;
 * the floor, every second row of quads at 6.8 TB/s, is 40). */
template <int DT, bool QUADS>
__global__ void __launch_bounds__(kHistThreads, 5)
    histogram_kernel(const uint8_t* __restrict__ pool, const HistJob* __restrict__ jobs,
                     const HistBrick K, uint32_t lanes_log2, uint32_t bin_copies_log2,
                     uint32_t n_bins, float lo, float scale_bins,
                     unsigned long long* __restrict__ per_brick,
                     unsigned long long* __restrict__ acc)
{
    extern __shared__ uint32_t counts[];
    const uint32_t copies_log2 = by_value(DT) ? kValueCopiesLog2 : bin_copies_log2;
    const uint32_t n_counts = (by_value(DT) ? 256u : n_bins) << copies_log2;
    for (uint32_t i = threadIdx.x; i < n_counts; i += kHistThreads)
        counts[i] = 0;
    __syncthreads();
    const HistJob job = jobs[blockIdx.x];
    const uint8_t* brick = pool + job.offset;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* mine = counts + (lane & ((1u << copies_log2) - 1u));
    auto count = [&](uint32_t bits) {
        const uint32_t k = by_value(DT) ? (bits & 255u)
                                        : bin_of(voxel_value<DT>(bits), lo, scale_bins, n_bins);
        atomicAdd(mine + (k << copies_log2), 1u);
    };
    constexpr uint32_t kStep = QUADS ? 2u : 1u; /* voxels a row or element stands for */
    const uint32_t ny = (K.B1 + kStep - 1u) / kStep, rows = ny * K.B2;
    const uint32_t per = (rows + gridDim.y - 1u) / gridDim.y;
    const uint32_t end = min(rows, (blockIdx.y + 1u) * per);
    const uint32_t stride = kHistWarps << (5u - lanes_log2);
    const uint32_t dy = stride % ny, dz = stride / ny;
    uint32_t row = blockIdx.y * per + (threadIdx.x >> lanes_log2);
    uint32_t y = row % ny, z = row / ny;
    const uint32_t x0 = kStep * (lane & ((1u << lanes_log2) - 1u));
    while (row < end)
    {
        uint32_t at[kHistRows], n = 0;
        bool up[kHistRows]; /* a second row of voxels in the row of quads */
#pragma unroll
        for (uint32_t u = 0; u < kHistRows; ++u)
            if (row < end)
            {
                up[u] = QUADS && 2u * y + 1u < K.B1;
                at[u] = ((z + K.O2) * K.N1 + kStep * y + K.O1) * K.N0 + K.O0;
                n = u + 1u;
                row += stride;
                y += dy;
                z += dz;
                if (y >= ny)
                {
                    y -= ny;
                    ++z;
                }
            }
        for (uint32_t x = x0; x < K.B0; x += kStep << lanes_log2)
        {
            uint32_t bits[kHistRows];
#pragma unroll
            for (uint32_t u = 0; u < kHistRows; ++u)
                if (u < n)
                    bits[u] = QUADS ? __ldg(reinterpret_cast<const uint32_t*>(brick) + at[u] + x)
                                    : load_voxel<DT>(brick, at[u] + x);
#pragma unroll
            for (uint32_t u = 0; u < kHistRows; ++u)
                if (u < n)
                {
                    count(bits[u]);
                    if (QUADS)
                    {
                        const bool right = x + 1u < K.B0;
                        if (right)
                            count(bits[u] >> 8);
                        if (up[u])
                            count(bits[u] >> 16);
                        if (right && up[u])
                            count(bits[u] >> 24);
                    }
                }
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < (by_value(DT) ? 256u : n_bins); k += kHistThreads)
    {
        unsigned long long c = 0;
        for (uint32_t i = 0; i < (1u << copies_log2); ++i)
            /* each thread starts at another copy: 32 banks */
            c += counts[(k << copies_log2) + ((i + k) & ((1u << copies_log2) - 1u))];
        if (c == 0)
            continue;
        c *= job.scale;
        const uint32_t b =
            by_value(DT) ? bin_of(voxel_value<DT>(k), lo, scale_bins, n_bins) : k;
        if (per_brick)
            atomicAdd(per_brick + uint64_t(blockIdx.x) * n_bins + b, c);
        atomicAdd(acc + b, c);
    }
}
} // namespace

extern "C" lv_status lv_histogram(lv_volume* vol, const uint64_t* ids, uint32_t n,
                                  uint32_t n_bins, float range_lo, float range_hi,
                                  uint64_t* per_brick, uint64_t* accumulated)
{
    if (!vol || (n && !ids) || !accumulated || n_bins < 2 || n_bins > 8192 ||
        !(range_hi > range_lo))
        return LV_EINVAL;
    lv_ctx* ctx = vol->ctx;
    std::lock_guard<std::mutex> lock(ctx->mutex);
    LV_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->upload_stream;
    std::fill(accumulated, accumulated + n_bins, uint64_t(0));
    if (n == 0)
        return LV_OK;
    /* the bricks must be resident: load the missing ones (nothing in flight
     * is protected beyond this call) */
    uint32_t loaded = 0;
    uint64_t bytes = 0;
    lv_status st = stream_bricks(ctx, vol, ids, n, ctx->renderer->frame + 1u, s, loaded, bytes);
    if (st != LV_OK)
        return st;
    /* the last call's kernel has read the jobs: each call waits for its own */
    PinnedBuffer& hjobs = ctx->renderer->h_hist_jobs;
    LV_CUDA(ctx, hjobs.reserve(sizeof(HistJob) * n));
    HistJob* jobs = hjobs.as<HistJob>();
    for (uint32_t i = 0; i < n; ++i)
    {
        const uint64_t id = ids[i];
        const uint32_t L = nid_level(id);
        if (L >= vol->info.depth)
            return fail(ctx, LV_EINVAL, "node id outside the volume");
        const uint64_t idx = node_index(vol->level_offset, vol->info.root_blocks, id);
        if (idx >= vol->n_nodes || vol->host_table[idx] < 0)
            return fail(ctx, LV_ENOTFOUND, "brick not resident (no data for the node)");
        const uint64_t side = uint64_t(1) << (vol->info.depth - 1u - L);
        jobs[i].offset = uint64_t(vol->host_table[idx]) * kSlotUnit;
        jobs[i].scale = side * side * side;
    }
    /* the accumulated counts, then the bricks', in a buffer the context keeps
     * up to kHistKeep bytes: allocating and freeing buffers on every call,
     * with a copy of the jobs, took 35 us (one brick: 59 -> 23 us a call) */
    const uint64_t out_bytes = sizeof(uint64_t) * n_bins * (per_brick ? uint64_t(n) + 1u : 1u);
    DeviceBuffer own_out;
    DeviceBuffer& dout = out_bytes <= kHistKeep ? ctx->renderer->hist_out : own_out;
    PinnedBuffer& hacc = ctx->renderer->h_hist_acc;
    LV_CUDA(ctx, dout.reserve(out_bytes));
    LV_CUDA(ctx, hacc.reserve(sizeof(uint64_t) * n_bins));
    LV_CUDA(ctx, cudaMemsetAsync(dout.ptr, 0, out_bytes, s));
    const float scale_bins = float(n_bins - 1) / (range_hi - range_lo);
    const auto& I = vol->info;
    const bool quads = vol->stage_off != 0;
    const HistBrick K{I.max_block[0], I.max_block[1], I.overlap[0], I.overlap[1], I.overlap[2],
                      I.max_block[0] - 2u * I.overlap[0], I.max_block[1] - 2u * I.overlap[1],
                      I.max_block[2] - 2u * I.overlap[2]};
    /* lanes to a row: the power of two that covers it, at most a warp */
    uint32_t lanes_log2 = 0;
    while (lanes_log2 < 5 && (quads ? 2u : 1u) << lanes_log2 < K.B0)
        ++lanes_log2;
    /* as many copies of the counters as fit, at most one per lane */
    const uint32_t counters = by_value(I.dtype) ? 256u : n_bins;
    uint32_t copies_log2 = 5;
    while (counters << copies_log2 > kHistCounters)
        --copies_log2;
    /* blocks of at least 64 rows */
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const uint64_t rows = uint64_t(K.B1) * K.B2;
    const uint32_t parts = uint32_t(std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t(sms) * kHistBlocksPerSm + n - 1) / n, rows / 64)));
    auto kernel = quads ? histogram_kernel<LV_DT_UINT8, true> : histogram_kernel<LV_DT_UINT8, false>;
    switch (I.dtype)
    {
    case LV_DT_UINT16: kernel = histogram_kernel<LV_DT_UINT16, false>; break;
    case LV_DT_INT8: kernel = histogram_kernel<LV_DT_INT8, false>; break;
    case LV_DT_INT16: kernel = histogram_kernel<LV_DT_INT16, false>; break;
    case LV_DT_UINT32: kernel = histogram_kernel<LV_DT_UINT32, false>; break;
    case LV_DT_INT32: kernel = histogram_kernel<LV_DT_INT32, false>; break;
    case LV_DT_FLOAT: kernel = histogram_kernel<LV_DT_FLOAT, false>; break;
    default: break;
    }
    kernel<<<dim3(n, std::min(parts, 65535u)), kHistThreads,
             sizeof(uint32_t) * (size_t(counters) << copies_log2), s>>>(
        ctx->pool->arena.as<uint8_t>(), hjobs.as_dev<HistJob>(), K, lanes_log2, copies_log2,
        n_bins, range_lo, scale_bins,
        per_brick ? dout.as<unsigned long long>() + n_bins : nullptr,
        dout.as<unsigned long long>());
    LV_CUDA(ctx, cudaGetLastError());
    LV_CUDA(ctx, cudaMemcpyAsync(hacc.ptr, dout.ptr, sizeof(uint64_t) * n_bins,
                                 cudaMemcpyDeviceToHost, s));
    /* the bricks' straight to the caller: through page-locked memory the host's
     * own copy of 1 MB cost more than it saved */
    if (per_brick)
        LV_CUDA(ctx, cudaMemcpyAsync(per_brick, dout.as<uint64_t>() + n_bins,
                                     sizeof(uint64_t) * n_bins * n, cudaMemcpyDeviceToHost, s));
    LV_CUDA(ctx, cudaStreamSynchronize(s));
    std::memcpy(accumulated, hacc.ptr, sizeof(uint64_t) * n_bins);
    return LV_OK;
}
