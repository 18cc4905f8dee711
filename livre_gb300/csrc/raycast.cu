/*
 * Residency resolve, leaf-grid build and the ray-cast kernel.
 *
 * Replaces the per-brick GL draw loop of livre/eq/render/RayCastRenderer.cpp
 * (onFrameRender :467-481, renderBrick :503-571) and the fragment shader
 * livre/eq/render/shaders/fragRayCast.glsl:113-207. Instead of one draw call
 * per brick with a read-modify-write of an RGBA32F image, one thread walks one
 * ray through every brick in ray order:
 *
 *  - the rendering set (visible bricks, or their nearest resident ancestors,
 *    RenderingSetGeneratorFilter.cpp:32-111) is splatted into a dense leaf
 *    grid at the finest octree level: one 32-bit entry per finest cell,
 *    (level << 27 | pool slot), coarser level winning;
 *  - samples lie on the global grid t = tnearGlobal + k * step, exactly the
 *    positions the shader's residue snapping produces (fragRayCast.glsl:
 *    142-147); a sample belongs to the brick whose cell contains it;
 *  - voxels are read straight from the HBM brick pool (nearest or trilinear,
 *    clamp to edge), mapped through the 1D transfer function (linear,
 *    clamp to edge) and composited front to back with the shader's opacity
 *    correction 1 - (1 - min(a, 255/256))^(32 / nSamples) and early exit.
 *
 * Ray geometry (direction, box and near-plane distances, sample positions,
 * cell and voxel coordinates) uses explicit IEEE round-to-nearest float
 * intrinsics in a fixed order, so every sample reads the same voxels as the
 * CPU oracle; shading runs in FP32 with fused multiply-adds.
 *
 * raycast_device.cuh holds the device code of a ray; this file the residency
 * and leaf-grid kernels, the kernels of uint8 and uint16 volumes with one lane
 * per ray and the dispatch; raycast_split.cu those with several lanes per ray
 * and raycast_types.cu those of the other voxel types.
 */
#include <algorithm>
#include <cmath>

#include "raycast_device.cuh"

namespace lv
{
namespace
{
/* Emits (id, slot) into the rendering set of the view. */
__device__ __forceinline__ void emit_render(const ResolveView& R, uint64_t id,
                                            uint32_t slot)
{
    const uint32_t k = atomicAdd(&R.counters[FC_RENDERED], 1u);
    if (k < R.render_capacity)
    {
        R.render_ids[k] = id;
        R.render_slots[k] = slot;
    }
    else
        atomicExch(&R.counters[FC_ERROR], 1u);
}

/* For each visible id: resident -> rendering set; missing -> missing list
 * and (async mode) the nearest resident ancestor, once per view. */
__device__ void resolve_body(const ResolveView& R, uint32_t first, uint32_t stride)
{
    const uint32_t n = *R.n_visible_ptr;
    for (uint32_t i = first; i < n; i += stride)
    {
        const uint64_t id = R.visible[i];
        const uint32_t L = nid_level(id);
        if (L >= R.depth || nid_x(id) >= (R.root_blocks[0] << L) ||
            nid_y(id) >= (R.root_blocks[1] << L) || nid_z(id) >= (R.root_blocks[2] << L))
        {
            atomicExch(&R.counters[FC_ERROR], 2u); /* id outside this octree */
            continue;
        }
        const uint64_t idx = node_index(R.level_offset, R.root_blocks, id);
        if (idx >= R.n_nodes)
        {
            atomicExch(&R.counters[FC_ERROR], 2u);
            continue;
        }
        const int32_t slot = R.node_table[idx];
        if (slot >= 0)
        {
            R.node_stamp[idx] = R.frame;
            R.view_stamp[idx] = R.view_frame;
            atomicAdd(&R.counters[FC_AVAILABLE], 1u);
            emit_render(R, id, uint32_t(slot));
            if (R.synchronous)
            {
                /* no ancestor fallback: the rendering set is part of the
                 * visible cut, nothing to prune */
                atomicAdd(&R.counters[FC_KEPT], 1u);
                atomicMax(&R.counters[FC_MAX_LEVEL], L + 1u);
            }
            continue;
        }
        atomicAdd(&R.counters[FC_NOT_AVAILABLE], 1u);
        const uint32_t m = atomicAdd(&R.counters[FC_MISSING], 1u);
        if (m < R.missing_capacity)
            R.missing[m] = id;
        if (R.synchronous)
            continue;
        uint64_t cur = id;
        while (nid_level(cur) > 0)
        {
            const uint32_t L = nid_level(cur) - 1u;
            cur = nid_make(L, nid_x(cur) >> 1, nid_y(cur) >> 1, nid_z(cur) >> 1,
                           nid_t(cur));
            const uint64_t pidx = node_index(R.level_offset, R.root_blocks, cur);
            const int32_t ps = R.node_table[pidx];
            if (ps >= 0)
            {
                /* the exchange comes first: on the single-view path the view
                 * stamps and the in-use stamps are the same array */
                if (atomicExch(&R.view_stamp[pidx], R.view_frame) != R.view_frame)
                    emit_render(R, cur, uint32_t(ps));
                R.node_stamp[pidx] = R.frame;
                break;
            }
        }
    }
}

/* A rendering-set entry that has an ancestor in the set: every entry of this
 * view carries view_stamp == view_frame. */
__device__ __forceinline__ bool shadowed(const ResolveView& R, uint64_t id)
{
    while (nid_level(id) > 0)
    {
        id = nid_make(nid_level(id) - 1u, nid_x(id) >> 1, nid_y(id) >> 1, nid_z(id) >> 1,
                      nid_t(id));
        if (R.view_stamp[node_index(R.level_offset, R.root_blocks, id)] == R.view_frame)
            return true;
    }
    return false;
}

/* Drops shadowed rendering-set entries, as
 * RenderingSetGenerator::generateRenderingSet does
 * (RenderingSetGeneratorFilter.cpp:63-79). */
__device__ void prune_body(const ResolveView& R, uint32_t first, uint32_t stride)
{
    const uint32_t n = min(R.counters[FC_RENDERED], R.render_capacity);
    for (uint32_t e = first; e < n; e += stride)
    {
        const uint64_t id = R.render_ids[e];
        if (shadowed(R, id))
            R.render_ids[e] = kInvalidNode;
        else
        {
            atomicAdd(&R.counters[FC_KEPT], 1u);
            atomicMax(&R.counters[FC_MAX_LEVEL], nid_level(id) + 1u);
        }
    }
}

/* The cells of the leaf grid under node id that fall to part `part` of
 * `parts`, dealt over the lanes of a warp. (A grid has at most 2^28 cells.) */
template <class F>
__device__ __forceinline__ void for_leaf_cells(const ResolveView& R, uint64_t id, uint32_t part,
                                               uint32_t parts, F&& f)
{
    const uint32_t sh = R.Lf - nid_level(id), mask = (1u << sh) - 1u, cells = 1u << (3u * sh);
    const uint32_t x0 = nid_x(id) << sh, y0 = nid_y(id) << sh, z0 = nid_z(id) << sh;
    for (uint32_t c = 32u * part + (threadIdx.x & 31u); c < cells; c += 32u * parts)
    {
        const uint32_t x = x0 + (c & mask), y = y0 + ((c >> sh) & mask), z = z0 + (c >> (2u * sh));
        if (x < R.dims[0] && y < R.dims[1] && z < R.dims[2])
            f((z * R.dims[1] + y) * R.dims[0] + x);
    }
}

/* Warps that share a node's cells where n nodes have nwarps warps: the fewer
 * nodes a frame renders, the more cells each covers. At most one per 256 cells,
 * so that a small grid is left to few warps. One warp for the 16.7 M cells
 * under the root of an 8192^3 octree in 32^3 bricks, shown small, made a frame
 * of 25.9 ms (asynchronous 38.6, with an atomic minimum per cell); shared it is
 * one of 86 us (93). The root of a 2048^3 octree in 64^3 bricks: 122 -> 71 us. */
__device__ __forceinline__ uint32_t cell_parts(const ResolveView& R, uint32_t n, uint32_t nwarps)
{
    const uint32_t chunks = (R.dims[0] * R.dims[1] * R.dims[2]) >> 8;
    return n && n < nwarps && n < chunks ? min(nwarps, chunks) / n : 1u;
}

/* Splats the rendering set into the leaf grid, a warp or several per entry. */
__device__ void leaf_fill_body(const ResolveView& R, uint32_t warp, uint32_t nwarps)
{
    const uint32_t n = min(R.counters[FC_RENDERED], R.render_capacity);
    const uint32_t parts = cell_parts(R, n, nwarps);
    for (uint32_t i = warp; i < n * parts; i += nwarps)
    {
        const uint32_t e = parts > 1u ? i % n : i;
        const uint64_t id = R.render_ids[e];
        if (id == kInvalidNode)
            continue;
        const uint32_t key =
            (nid_level(id) << kLeafSlotBits) | (R.render_slots[e] & kLeafSlotMask);
        for_leaf_cells(R, id, parts > 1u ? i / n : 0u, parts,
                       [&](uint32_t cell) { atomicMin(&R.leaf[cell], key); });
    }
}

/* The residency pass of one view, a warp or several per visible node
 * (resolve_body's rules).
 *
 * SYNC: no ancestor fallback. The rendering set is part of the visible cut,
 * whose nodes do not overlap, so the nodes' cells of the leaf grid are simply
 * stored (cell_parts), and the last block to finish writes the counters, the
 * selection's words and the missing ids into mapped page-locked host memory,
 * where the host waits for them. Else a missing node's nearest resident
 * ancestor is emitted, prune_leaf_kernel drops the entries it shadows and
 * stores the others' cells, and only the selection's words go to the host.
 *
 * The synchronous pass used to be three launches (resolve, read-back, leaf
 * fill), behind one for the selection's words and a clear of the counters:
 * frames of a 100^3 volume 63.1 -> 54.9 us, of a 256^3 one at 512 x 512
 * 141 -> 134. */
template <bool SYNC>
__global__ void __launch_bounds__(256)
    residency_kernel(const __grid_constant__ ResolveView R, const uint32_t* __restrict__ sel_words,
                     uint32_t* h_words, uint64_t* h_missing)
{
    __shared__ uint32_t available, missing, max_level, error, last;
    if (threadIdx.x == 0)
        available = missing = max_level = error = 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n = *R.n_visible_ptr;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t parts = SYNC ? cell_parts(R, n, nwarps) : 1u;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n * parts; i += nwarps)
    {
        const uint32_t part = parts > 1u ? i / n : 0u;
        const bool lead = lane == 0 && part == 0; /* reports the node */
        uint64_t id = R.visible[i - part * n];
        uint32_t L = nid_level(id);
        const bool inside = L < R.depth && nid_x(id) < (R.root_blocks[0] << L) &&
                            nid_y(id) < (R.root_blocks[1] << L) &&
                            nid_z(id) < (R.root_blocks[2] << L);
        const uint64_t idx =
            inside ? node_index(R.level_offset, R.root_blocks, id) : R.n_nodes;
        if (idx >= R.n_nodes)
        {
            error = 2u; /* id outside this octree */
            continue;
        }
        int32_t slot = R.node_table[idx];
        if (slot >= 0)
        {
            if (lead)
            {
                R.node_stamp[idx] = R.frame;
                R.view_stamp[idx] = R.view_frame;
                atomicAdd(&available, 1u);
                if (SYNC)
                    atomicMax(&max_level, L + 1u);
                emit_render(R, id, uint32_t(slot));
            }
        }
        else
        {
            if (lead)
            {
                atomicAdd(&missing, 1u);
                const uint32_t m = atomicAdd(&R.counters[FC_MISSING], 1u);
                if (m < R.missing_capacity)
                    R.missing[m] = id;
            }
            if (SYNC)
                continue;
            /* the nearest resident ancestor, emitted once per view (the same
             * walk in every lane) */
            while (slot < 0 && L > 0)
            {
                --L;
                id = nid_make(L, nid_x(id) >> 1, nid_y(id) >> 1, nid_z(id) >> 1, nid_t(id));
                slot = R.node_table[node_index(R.level_offset, R.root_blocks, id)];
            }
            if (slot >= 0 && lane == 0)
            {
                const uint64_t p = node_index(R.level_offset, R.root_blocks, id);
                /* the exchange comes first: the view stamps and the in-use
                 * stamps may be the same array */
                if (atomicExch(&R.view_stamp[p], R.view_frame) != R.view_frame)
                    emit_render(R, id, uint32_t(slot));
                R.node_stamp[p] = R.frame;
            }
        }
        if (SYNC)
        {
            const uint32_t key = (L << kLeafSlotBits) | (uint32_t(slot) & kLeafSlotMask);
            for_leaf_cells(R, id, part, parts, [&](uint32_t cell) { R.leaf[cell] = key; });
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (available)
        {
            atomicAdd(&R.counters[FC_AVAILABLE], available);
            if (SYNC)
            {
                atomicAdd(&R.counters[FC_KEPT], available);
                atomicMax(&R.counters[FC_MAX_LEVEL], max_level);
            }
        }
        if (missing)
            atomicAdd(&R.counters[FC_NOT_AVAILABLE], missing);
        if (error)
            atomicExch(&R.counters[FC_ERROR], error);
        if (SYNC)
        {
            __threadfence();
            last = atomicAdd(&R.counters[FC_TICKET], 1u) == gridDim.x - 1u;
        }
        else
            last = blockIdx.x == 0;
    }
    __syncthreads();
    if (!last)
        return;
    if (threadIdx.x < LV_SELECT_RESULT_WORDS)
        h_words[FC_WORDS + threadIdx.x] = sel_words[threadIdx.x];
    if (SYNC)
    {
        __threadfence();
        if (threadIdx.x < FC_WORDS)
            h_words[threadIdx.x] = __ldcg(R.counters + threadIdx.x);
        const uint32_t n_ids = min(__ldcg(R.counters + FC_MISSING), R.missing_capacity);
        for (uint32_t i = threadIdx.x; i < n_ids; i += blockDim.x)
            h_missing[i] = __ldcg(R.missing + i);
    }
    __threadfence_system();
}

/* The end of an asynchronous residency pass, a warp or several per entry of
 * the rendering set: drops the entry if it is shadowed, else counts it and
 * stores its cells of the leaf grid (the entries kept do not overlap). A warp
 * that finds the entry dropped already leaves it; one that does not comes to
 * the same answer. */
__global__ void __launch_bounds__(256)
    prune_leaf_kernel(const __grid_constant__ ResolveView R)
{
    __shared__ uint32_t kept, max_level;
    if (threadIdx.x == 0)
        kept = max_level = 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n = min(R.counters[FC_RENDERED], R.render_capacity);
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5, parts = cell_parts(R, n, nwarps);
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n * parts; i += nwarps)
    {
        const uint32_t part = parts > 1u ? i / n : 0u, e = i - part * n;
        const bool lead = lane == 0 && part == 0;
        const uint64_t id = *static_cast<volatile uint64_t*>(R.render_ids + e);
        if (__any_sync(0xFFFFFFFFu, id == kInvalidNode))
            continue;
        if (shadowed(R, id))
        {
            if (lead)
                R.render_ids[e] = kInvalidNode;
            continue;
        }
        const uint32_t L = nid_level(id);
        if (lead)
        {
            atomicAdd(&kept, 1u);
            atomicMax(&max_level, L + 1u);
        }
        const uint32_t key = (L << kLeafSlotBits) | (R.render_slots[e] & kLeafSlotMask);
        for_leaf_cells(R, id, part, parts, [&](uint32_t cell) { R.leaf[cell] = key; });
    }
    __syncthreads();
    if (threadIdx.x == 0 && kept)
    {
        atomicAdd(&R.counters[FC_KEPT], kept);
        atomicMax(&R.counters[FC_MAX_LEVEL], max_level);
    }
}

__global__ void resolve_kernel(ResolveView R)
{
    resolve_body(R, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
/* multi-view variants: blockIdx.y selects the view */
__global__ void resolve_views_kernel(const ResolveView* __restrict__ Rs)
{
    resolve_body(Rs[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x,
                 gridDim.x * blockDim.x);
}
__global__ void prune_views_kernel(const ResolveView* __restrict__ Rs)
{
    prune_body(Rs[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x,
               gridDim.x * blockDim.x);
}
__global__ void leaf_fill_views_kernel(const ResolveView* __restrict__ Rs)
{
    leaf_fill_body(Rs[blockIdx.y], (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                   (gridDim.x * blockDim.x) >> 5);
}

/* nSamplesPerRay from the finest rendered level (RayCastRenderer.cpp:
 * 216-233 for LV_STEP_REFERENCE; half a voxel for LV_STEP_HALF_VOXEL). */
__device__ void step_body(uint32_t* counters, uint32_t fixed, uint32_t policy,
                          uint32_t max_voxel_dim, uint32_t depth)
{
    uint32_t n = fixed;
    if (n == 0)
    {
        const uint32_t ml = counters[FC_MAX_LEVEL];
        const uint32_t L = ml ? ml - 1u : 0u;
        const uint32_t shift = depth - L - 1u;
        if (policy == LV_STEP_HALF_VOXEL)
            n = (2u * max_voxel_dim) >> shift;
        else
        {
            const float at_lod = float(max_voxel_dim) / float(1u << shift);
            n = uint32_t(fmaxf(at_lod, 512.0f));
        }
        if (n == 0)
            n = 1;
    }
    counters[FC_SAMPLES_PER_RAY] = n;
}

__global__ void step_views_kernel(const RayView* __restrict__ views, uint32_t n)
{
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n)
        step_body(views[v].counters, views[v].samples_fixed, views[v].step_policy,
                  views[v].max_voxel_dim, views[v].depth);
}

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

/* LA: one-sample look-ahead */
template <int DT, int FILTER, int EDGE, int LA>
__global__ void __launch_bounds__(256) raycast_kernel(const RayView V)
{
    if (skip_frame(V))
        return;
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t py = blockIdx.y * blockDim.y + threadIdx.y;
    const uint32_t n = frame_samples(V);
    const float step = __fdiv_rn(1.0f, __uint2float_rn(n));
    const float ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    uint32_t nsamp = 0;
    if (px < V.W && py < V.H)
    {
        const RayGeom g = ray_setup(V, px, py);
        const float4 r =
            march<DT, FILTER, 0, EDGE, LA>(V, V, g, step, ac, nsamp, initial_dst(V, px, py));
        V.out[frame_index(V, px, py)] = r;
    }
    /* warp-aggregated 64-bit sample count */
    unsigned long long s = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_down_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x + threadIdx.y * blockDim.x) % 32 == 0 && s)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), s);
}

/* Batched mode: one persistent launch renders the tiles of many views. Each
 * CTA pops (view, tile) work items from a device queue (one atomic per
 * tile), keeps the current view's constants (and optionally its transfer
 * function) in shared memory, and ray casts tile_w x tile_h pixels. */
template <int DT, int FILTER, int TF_SHARED, int EDGE>
__global__ void __launch_bounds__(256)
    raycast_persistent_kernel(const RayView* __restrict__ views, TileQueue Q)
{
    __shared__ RayView sV;
    __shared__ uint32_t s_item, s_view;
    extern __shared__ float4 s_tf[];
    const uint32_t n_views = *Q.n_views;
    const uint32_t total = Q.tile_start[n_views];
    if (threadIdx.x == 0)
        atomicCAS(Q.clock, 0ull, globaltimer());
    uint32_t cached = 0xFFFFFFFFu;
    float step = 0.f, ac = 0.f;
    HotView H{};
    for (;;)
    {
        if (threadIdx.x == 0)
        {
            uint32_t item = atomicAdd(Q.head, 1u);
            if (Q.order && item < total)
                item = Q.order[item];
            uint32_t lo = 0, hi = n_views;
            if (item < total)
                while (hi - lo > 1)
                {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (Q.tile_start[mid] <= item)
                        lo = mid;
                    else
                        hi = mid;
                }
            s_item = item;
            s_view = lo;
        }
        __syncthreads();
        const uint32_t item = s_item;
        const uint32_t gv = s_view;
        if (item >= total)
            break;
        const uint32_t v = Q.view_ids[gv];
        if (v != cached)
        {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(views + v);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&sV);
            for (uint32_t w = threadIdx.x; w < sizeof(RayView) / 4; w += blockDim.x)
                dst[w] = src[w];
            __syncthreads();
            if (TF_SHARED)
            {
                for (uint32_t i = threadIdx.x; i < 2u * sV.tfn; i += blockDim.x)
                    s_tf[i] = sV.tf[i];
                __syncthreads();
                if (threadIdx.x == 0)
                    sV.tf = s_tf;
                __syncthreads();
            }
            cached = v;
            H = hot_view(sV);
            const uint32_t n = sV.counters[FC_SAMPLES_PER_RAY];
            step = __fdiv_rn(1.0f, __uint2float_rn(n));
            ac = __fdiv_rn(32.0f, __uint2float_rn(n));
        }
        const uint32_t t = item - Q.tile_start[gv];
        const uint32_t tiles_x = (sV.W + Q.tile_w - 1) / Q.tile_w;
        const uint32_t px = (t % tiles_x) * Q.tile_w + threadIdx.x % Q.tile_w;
        const uint32_t py = (t / tiles_x) * Q.tile_h + threadIdx.x / Q.tile_w;
        uint32_t nsamp = 0;
        if (px < sV.W && py < sV.H && threadIdx.x < Q.tile_w * Q.tile_h)
        {
            const RayGeom g = ray_setup(sV, px, py);
            const float4 r = march<DT, FILTER, TF_SHARED, EDGE, 0>(sV, H, g, step, ac, nsamp);
            sV.out[frame_index(sV, px, py)] = r;
        }
        unsigned long long sum = nsamp;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
        if ((threadIdx.x & 31u) == 0 && sum)
            atomicAdd(reinterpret_cast<unsigned long long*>(sV.counters + FC_SAMPLES_LO), sum);
        __syncthreads();
    }
    if (threadIdx.x == 0)
        atomicMax(Q.clock + 1, globaltimer());
}

/* Longest-first tile order of one view. A tile's cost is estimated by the
 * length of its centre ray inside the volume (near and clip planes
 * applied), quantised to kTileBuckets classes; a counting sort lists the
 * longest class first (the order within a class does not matter: every
 * pixel is computed independently). hist[0, kTileBuckets) are the class
 * counts and hist[kTileBuckets, 2 kTileBuckets) the scatter cursors, both
 * zeroed before the key pass. */
constexpr uint32_t kTileBuckets = 64;

/* Slot of an item of class `key` in the sorted order: the class's first
 * slot (base, shared memory) plus the item's rank among the class's items
 * claimed so far, one global atomic per class present in the warp (items of
 * one class are many: per-item atomics on one cursor serialised). key =
 * kTileBuckets: no item (the lane still takes part in the warp-wide
 * match). */
__device__ __forceinline__ uint32_t base_of_item(const uint32_t* base, uint32_t* hist,
                                                 uint32_t key)
{
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t leader = __ffs(peers) - 1u;
    uint32_t first = 0;
    if (lane == leader && key < kTileBuckets)
        first = atomicAdd(&hist[kTileBuckets + key], __popc(peers));
    first = __shfl_sync(0xFFFFFFFFu, first, leader); /* each lane: its class's leader */
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    return key < kTileBuckets ? base[key] + first + rank : 0xFFFFFFFFu;
}

__global__ void __launch_bounds__(256)
    tile_key_kernel(const RayView V, uint32_t tile_w, uint32_t tile_h, uint32_t tiles_x,
                    uint32_t total, float buckets_per_length, uint8_t* __restrict__ keys,
                    uint32_t* __restrict__ hist)
{
    __shared__ uint32_t h[kTileBuckets];
    for (uint32_t i = threadIdx.x; i < kTileBuckets; i += blockDim.x)
        h[i] = 0;
    __syncthreads();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < total)
    {
        const uint32_t px = min((t % tiles_x) * tile_w + tile_w / 2, V.W - 1);
        const uint32_t py = min((t / tiles_x) * tile_h + tile_h / 2, V.H - 1);
        const RayGeom g = ray_setup(V, px, py);
        const float len = g.hit && g.tlo <= g.thi ? g.thi - g.tlo : 0.0f;
        const uint32_t q = uint32_t(fminf(len * buckets_per_length, float(kTileBuckets - 1)));
        const uint32_t key = kTileBuckets - 1u - q;
        keys[t] = uint8_t(key);
        atomicAdd(&h[key], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kTileBuckets; i += blockDim.x)
        if (h[i])
            atomicAdd(&hist[i], h[i]);
}

__global__ void __launch_bounds__(256)
    tile_order_kernel(const uint8_t* __restrict__ keys, uint32_t* __restrict__ hist,
                      uint32_t* __restrict__ order, uint32_t total)
{
    __shared__ uint32_t base[kTileBuckets];
    /* class counts loaded in parallel, then one thread scans them in shared
     * memory (a serial scan over global memory cost ~14 us per launch) */
    if (threadIdx.x < kTileBuckets)
        base[threadIdx.x] = hist[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t acc = 0;
        for (uint32_t k = 0; k < kTileBuckets; ++k)
        {
            const uint32_t c = base[k];
            base[k] = acc;
            acc += c;
        }
    }
    __syncthreads();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t key = t < total ? keys[t] : kTileBuckets;
    const uint32_t pos = base_of_item(base, hist, key);
    if (t < total && pos < total)
        order[pos] = t;
}

/* Single view on a resident grid: CTAs take tile_w x tile_h pixel tiles
 * (one ray per thread) from a device queue, the view's FC_QUEUE counter. */
template <int DT, int FILTER, int EDGE, int LA>
__global__ void __launch_bounds__(256)
    raycast_queue_kernel(const RayView V, uint32_t tile_w, uint32_t tile_h,
                         const uint32_t* __restrict__ order)
{
    if (skip_frame(V))
        return;
    __shared__ uint32_t s_item;
    const uint32_t n = frame_samples(V);
    const float step = __fdiv_rn(1.0f, __uint2float_rn(n));
    const float ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    const uint32_t tiles_x = (V.W + tile_w - 1) / tile_w;
    const uint32_t total = tiles_x * ((V.H + tile_h - 1) / tile_h);
    const uint32_t tx = threadIdx.x % tile_w, ty = threadIdx.x / tile_w;
    uint32_t nsamp = 0;
    for (;;)
    {
        if (threadIdx.x == 0)
            s_item = atomicAdd(V.counters + FC_QUEUE, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        __syncthreads();
        if (item >= total)
            break;
        const uint32_t tile = order ? order[item] : item;
        const uint32_t px = (tile % tiles_x) * tile_w + tx;
        const uint32_t py = (tile / tiles_x) * tile_h + ty;
        if (px < V.W && py < V.H)
        {
            const RayGeom g = ray_setup(V, px, py);
            V.out[frame_index(V, px, py)] =
                march<DT, FILTER, 0, EDGE, LA>(V, V, g, step, ac, nsamp, initial_dst(V, px, py));
        }
    }
    unsigned long long sum = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31u) == 0 && sum)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), sum);
}

/* Resident grid, warp-granular queue: each warp pops a 32-pixel tile (one
 * ray per lane) from the view's FC_QUEUE counter, in the given order. */
template <int DT, int FILTER, int EDGE, int LA>
__global__ void __launch_bounds__(128)
    raycast_warp_tiles_kernel(const RayView V, uint32_t tile_w, uint32_t tile_h,
                              const uint32_t* __restrict__ order)
{
    if (skip_frame(V))
        return;
    const uint32_t n = frame_samples(V);
    const float step = __fdiv_rn(1.0f, __uint2float_rn(n));
    const float ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    const uint32_t tiles_x = (V.W + tile_w - 1) / tile_w;
    const uint32_t total = tiles_x * ((V.H + tile_h - 1) / tile_h);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t nsamp = 0;
    for (;;)
    {
        uint32_t item = 0;
        if (lane == 0)
            item = atomicAdd(V.counters + FC_QUEUE, 1u);
        item = __shfl_sync(0xFFFFFFFFu, item, 0);
        if (item >= total)
            break;
        const uint32_t tile = order ? order[item] : item;
        const uint32_t px = (tile % tiles_x) * tile_w + lane % tile_w;
        const uint32_t py = (tile / tiles_x) * tile_h + lane / tile_w;
        if (px < V.W && py < V.H)
        {
            const RayGeom g = ray_setup(V, px, py);
            V.out[frame_index(V, px, py)] =
                march<DT, FILTER, 0, EDGE, LA>(V, V, g, step, ac, nsamp, initial_dst(V, px, py));
        }
        __syncwarp();
    }
    unsigned long long sum = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0 && sum)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), sum);
}

/* ---------------------------------------------------------------- refill
 * Persistent ray cast with lane refill. Every warp takes tile_w x tile_h
 * pixel tiles from a device queue (one atomic per tile) and hands the tile's
 * pixels to its lanes in order; a lane whose ray has finished takes the next
 * pixel at the next check (every `checks` samples), so lanes do not idle
 * while the longest ray of their warp finishes. When a tile runs out, the
 * warp takes the next one of the same view without waiting for its lanes;
 * a tile of another view (batched launch) is started once the warp has
 * drained. Each ray takes exactly the samples of march() in the same
 * order, so the image is identical to the one-thread-per-pixel kernel's. */
constexpr uint32_t kRefillThreads = 128;
constexpr uint32_t kRefillMinCtas = 8; /* 32 warps per SM: at most 64 registers */
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kNoItem = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t warp_pop(uint32_t* head)
{
    uint32_t v = 0;
    if ((threadIdx.x & 31u) == 0)
        v = atomicAdd(head, 1u);
    return __shfl_sync(kFull, v, 0);
}

/* group view of a work item: tile_start is ascending, tile_start[0] = 0 */
__device__ __forceinline__ uint32_t find_view(const TileQueue& Q, uint32_t n_views,
                                              uint32_t item)
{
    uint32_t lo = 0, hi = n_views;
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) >> 1;
        if (Q.tile_start[mid] <= item)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void load_view(RayView* dst, const RayView* src)
{
    __syncwarp();
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(dst);
    for (uint32_t w = threadIdx.x & 31u; w < sizeof(RayView) / 4; w += 32)
        d[w] = s[w];
    __syncwarp();
}

/* Longest-first order of the work items of one batched group. The cost of
 * a (view, tile) item is estimated as the samples of the tile's centre ray,
 * its length inside the volume times the view's samples per unit length,
 * in classes of a quarter octave; a counting sort lists the costliest
 * class first. hist holds the class counts then the scatter cursors, both
 * zeroed before the key pass. */
__global__ void __launch_bounds__(256)
    batch_key_kernel(const RayView* __restrict__ views, TileQueue Q, uint8_t* __restrict__ keys,
                     uint32_t* __restrict__ hist)
{
    __shared__ uint32_t h[kTileBuckets];
    for (uint32_t i = threadIdx.x; i < kTileBuckets; i += blockDim.x)
        h[i] = 0;
    __syncthreads();
    const uint32_t n_views = *Q.n_views;
    const uint32_t total = Q.tile_start[n_views];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += gridDim.x * blockDim.x)
    {
        const uint32_t gv = find_view(Q, n_views, i);
        const RayView& V = views[Q.view_ids[gv]];
        const uint32_t tile = i - Q.tile_start[gv];
        const uint32_t tiles_x = (V.W + Q.tile_w - 1) / Q.tile_w;
        const uint32_t px = min((tile % tiles_x) * Q.tile_w + Q.tile_w / 2, V.W - 1);
        const uint32_t py = min((tile / tiles_x) * Q.tile_h + Q.tile_h / 2, V.H - 1);
        const RayGeom g = ray_setup(V, px, py);
        const float len = g.hit && g.tlo <= g.thi ? g.thi - g.tlo : 0.0f;
        const float est = len * __uint2float_rn(V.counters[FC_SAMPLES_PER_RAY]);
        const uint32_t q = uint32_t(fminf(log2f(est + 1.0f) * 4.0f, float(kTileBuckets - 1)));
        const uint32_t key = kTileBuckets - 1u - q;
        keys[i] = uint8_t(key);
        atomicAdd(&h[key], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kTileBuckets; i += blockDim.x)
        if (h[i])
            atomicAdd(&hist[i], h[i]);
}

__global__ void __launch_bounds__(256)
    batch_order_kernel(TileQueue Q, const uint8_t* __restrict__ keys,
                       uint32_t* __restrict__ hist, uint32_t* __restrict__ order)
{
    __shared__ uint32_t base[kTileBuckets];
    /* class counts loaded in parallel, then one thread scans them in shared
     * memory (a serial scan over global memory cost ~14 us per launch) */
    if (threadIdx.x < kTileBuckets)
        base[threadIdx.x] = hist[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t acc = 0;
        for (uint32_t k = 0; k < kTileBuckets; ++k)
        {
            const uint32_t c = base[k];
            base[k] = acc;
            acc += c;
        }
    }
    __syncthreads();
    const uint32_t total = Q.tile_start[*Q.n_views];
    /* warp-uniform trip count: every lane reaches the warp-wide match */
    for (uint32_t b0 = blockIdx.x * blockDim.x; b0 < total; b0 += gridDim.x * blockDim.x)
    {
        const uint32_t i = b0 + threadIdx.x;
        const uint32_t key = i < total ? keys[i] : kTileBuckets;
        const uint32_t pos = base_of_item(base, hist, key);
        if (i < total && pos < total)
            order[pos] = i;
    }
}

__device__ __forceinline__ void flush_samples(const RayView& V, uint32_t nsamp)
{
    unsigned long long s = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_down_sync(kFull, s, o);
    if ((threadIdx.x & 31u) == 0 && s)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), s);
}

struct ViewConsts
{
    float step, ac;
    uint32_t tiles_x;
};

__device__ __forceinline__ ViewConsts view_consts(const RayView& V, uint32_t tile_w)
{
    ViewConsts k;
    const uint32_t n = view_samples(V);
    k.step = __fdiv_rn(1.0f, __uint2float_rn(n));
    k.ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    k.tiles_x = (V.W + tile_w - 1) / tile_w;
    return k;
}

/* MULTI: V is this warp's shared copy `sv` of the current view, reloaded
 * from `views` on a view change; else V is the launch's single view. */
template <int DT, int FILTER, int EDGE, bool MULTI>
__device__ __forceinline__ void refill_body(const RayView& V, RayView* sv,
                                            const RayView* __restrict__ views,
                                            const TileQueue& Q, uint32_t* head,
                                            uint32_t n_views, uint32_t total, uint32_t checks,
                                            const uint32_t* __restrict__ order)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t tw = Q.tile_w, th = Q.tile_h, npix = tw * th;
    uint32_t item = warp_pop(head);
    if (item >= total)
        return;
    uint32_t gv = 0;
    if (MULTI)
    {
        gv = find_view(Q, n_views, item);
        load_view(sv, views + Q.view_ids[gv]);
    }
    ViewConsts K = view_consts(V, tw);
    uint32_t tile = MULTI ? item - Q.tile_start[gv] : (order ? order[item] : item);
    uint32_t next = 0, pending = kNoItem;
    bool exhausted = false, active = false;
    uint32_t px = 0, py = 0, nsamp = 0;
    RayState r;
    for (;;)
    {
        /* hand the tile's next pixels to idle lanes, in lane order */
        for (;;)
        {
            const uint32_t idle = __ballot_sync(kFull, !active);
            if (!idle)
                break;
            if (next >= npix)
            {
                if (exhausted || pending != kNoItem)
                    break;
                const uint32_t nitem = warp_pop(head);
                if (nitem >= total)
                {
                    exhausted = true;
                    break;
                }
                if (MULTI && find_view(Q, n_views, nitem) != gv)
                {
                    pending = nitem; /* another view: drain first */
                    break;
                }
                tile = MULTI ? nitem - Q.tile_start[gv] : (order ? order[nitem] : nitem);
                next = 0;
            }
            const uint32_t mine = next + __popc(idle & below);
            next = min(next + uint32_t(__popc(idle)), npix);
            if (!active && mine < npix)
            {
                px = (tile % K.tiles_x) * tw + mine % tw;
                py = (tile / K.tiles_x) * th + mine / tw;
                if (px < V.W && py < V.H)
                {
                    const RayGeom g = ray_setup(V, px, py);
                    const float4 init = initial_dst(V, px, py);
                    active = ray_begin(g, K.step, r) && !(init.w > V.early);
                    r.dst = init;
                    if (!active)
                        V.out[frame_index(V, px, py)] = init;
                }
            }
        }
        if (!__any_sync(kFull, active))
        {
            if (MULTI && pending != kNoItem)
            {
                flush_samples(V, nsamp);
                nsamp = 0;
                gv = find_view(Q, n_views, pending);
                load_view(sv, views + Q.view_ids[gv]);
                K = view_consts(V, tw);
                tile = pending - Q.tile_start[gv];
                pending = kNoItem;
                next = 0;
                continue;
            }
            break; /* queue exhausted and every lane done */
        }
        if (active)
            for (uint32_t k = 0; k < checks; ++k)
                if (!ray_step<DT, FILTER, 0, EDGE>(V, V, r, K.step, K.ac, nsamp))
                {
                    active = false;
                    V.out[frame_index(V, px, py)] = r.dst;
                    flush_error(V, r);
                    break;
                }
    }
    flush_samples(V, nsamp);
}

/* Single view (lv_render): the queue head is the view's FC_QUEUE counter. */
template <int DT, int FILTER, int EDGE>
__global__ void __launch_bounds__(kRefillThreads, kRefillMinCtas)
    raycast_refill_kernel(const RayView V, uint32_t tile_w, uint32_t tile_h, uint32_t checks,
                          const uint32_t* __restrict__ order)
{
    if (skip_frame(V))
        return;
    TileQueue Q{};
    Q.tile_w = tile_w;
    Q.tile_h = tile_h;
    frame_samples(V);
    const uint32_t tiles = ((V.W + tile_w - 1) / tile_w) * ((V.H + tile_h - 1) / tile_h);
    refill_body<DT, FILTER, EDGE, false>(V, nullptr, nullptr, Q, V.counters + FC_QUEUE, 1u,
                                         tiles, checks, order);
}

/* Batched: tiles of many views of one kernel variant. */
template <int DT, int FILTER, int EDGE>
__global__ void __launch_bounds__(kRefillThreads, kRefillMinCtas)
    raycast_refill_views_kernel(const RayView* __restrict__ views, TileQueue Q, uint32_t checks)
{
    __shared__ RayView sV[kRefillThreads / 32];
    if (threadIdx.x == 0)
        atomicCAS(Q.clock, 0ull, globaltimer());
    const uint32_t n_views = *Q.n_views;
    RayView* sv = sV + (threadIdx.x >> 5);
    refill_body<DT, FILTER, EDGE, true>(*sv, sv, views, Q, Q.head, n_views,
                                        Q.tile_start[n_views], checks, nullptr);
    if ((threadIdx.x & 31u) == 0)
        atomicMax(Q.clock + 1, globaltimer());
}

/* Pixels of the frame a launch clears: the rect [x0, x0 + W) x [y0, y0 + H)
 * without [ix0, ix1) x [iy0, iy1). */
struct ClearRect
{
    float4* out;
    uint32_t FW, x0, y0, W, H, ix0, iy0, ix1, iy1;
};

/* Transparent black in the pixels of C. */
__device__ __forceinline__ void clear_pixels(const ClearRect& C)
{
    for (uint32_t y = C.y0 + blockIdx.y; y < C.y0 + C.H; y += gridDim.y)
    {
        const bool row = y >= C.iy0 && y < C.iy1;
        for (uint32_t x = C.x0 + blockIdx.x * blockDim.x + threadIdx.x; x < C.x0 + C.W;
             x += gridDim.x * blockDim.x)
            if (!(row && x >= C.ix0 && x < C.ix1))
                C.out[uint64_t(y) * C.FW + x] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__global__ void __launch_bounds__(256) clear_outside_kernel(const ClearRect C) { clear_pixels(C); }

/* What a frame clears before its residency pass, in one launch instead of a
 * clear each: its counters, the leaf grid, and the pixels of C (W = 0: none).
 * A small frame is bound by the host's calls, about 1.7 us each: with this,
 * no clear for the selection of a small octree, no tile order where all tiles
 * are resident and one event in place of two, twice, a frame makes 23 instead
 * of 33, and one of a 100^3 volume takes 49.4 us (56.3). */
__global__ void __launch_bounds__(256)
    frame_clear_kernel(uint32_t* __restrict__ counters, uint32_t* __restrict__ leaf,
                       uint64_t cells, const ClearRect C)
{
    const uint64_t t = (uint64_t(blockIdx.y) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < FC_WORDS)
        counters[t] = 0u;
    /* four cells a store: the grid is a device allocation */
    const uint64_t threads = uint64_t(gridDim.x) * gridDim.y * blockDim.x;
    for (uint64_t i = t; i < cells / 4u; i += threads)
        reinterpret_cast<uint4*>(leaf)[i] =
            make_uint4(kLeafEmpty, kLeafEmpty, kLeafEmpty, kLeafEmpty);
    if (t < (cells & 3u))
        leaf[(cells & ~uint64_t(3)) + t] = kLeafEmpty;
    if (C.W)
        clear_pixels(C);
}

__global__ void to_rgba8_kernel(const float4* __restrict__ in,
                                uchar4* __restrict__ out, uint64_t n)
{
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
         i += uint64_t(gridDim.x) * blockDim.x)
    {
        const float4 c = in[i];
        const auto q = [](float v) {
            return (unsigned char)(fminf(fmaxf(v, 0.0f), 1.0f) * 255.0f);
        };
        out[i] = make_uchar4(q(c.x), q(c.y), q(c.z), 255);
    }
}

} // namespace

lv_status launch_resolve(lv_ctx* ctx, const ResolveView& R, cudaStream_t s)
{
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    resolve_kernel<<<sms, 256, 0, s>>>(R);
    ++ctx->kernels;
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

lv_status launch_residency(lv_ctx* ctx, const ResolveView& R, const uint32_t* sel_words,
                           uint32_t* h_words, uint64_t* h_missing, cudaStream_t s)
{
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (R.synchronous)
        residency_kernel<true><<<sms, 256, 0, s>>>(R, sel_words, h_words, h_missing);
    else
    {
        residency_kernel<false><<<sms, 256, 0, s>>>(R, sel_words, h_words, h_missing);
        LV_CUDA(ctx, cudaGetLastError());
        prune_leaf_kernel<<<sms, 256, 0, s>>>(R);
        ++ctx->kernels;
    }
    ++ctx->kernels;
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

namespace
{
/* CTAs of `kernel` resident on the whole GPU at once (occupancy API). */
template <typename K>
uint32_t resident_ctas(lv_ctx* ctx, K kernel, int threads, size_t smem, int most = 32)
{
    int per_sm = 0, sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
            cudaSuccess ||
        per_sm < 1)
    {
        cudaGetLastError();
        per_sm = 1;
    }
    return uint32_t(std::min(per_sm, most)) * uint32_t(sms);
}

/* One instantiation per (voxel type, filter, TF staging, edge clamping);
 * ctas = 0: as many CTAs as are resident at once. */
template <int DT, int F, int TFS, int EDGE>
lv_status persistent_dispatch(lv_ctx* ctx, const RayView* d_rays, const TileQueue& Q,
                              uint32_t ctas, size_t smem, cudaStream_t s)
{
    auto k = raycast_persistent_kernel<DT, F, TFS, EDGE>;
    if (smem > 48 * 1024)
        LV_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(smem)));
    const int threads = int(Q.tile_w * Q.tile_h);
    uint32_t grid = resident_ctas(ctx, k, threads, smem);
    if (ctas)
    {
        int sms = 152;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        grid = uint32_t(sms) * ctas;
    }
    k<<<grid, threads, smem, s>>>(d_rays, Q);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

template <int DT, int F, int EDGE>
lv_status refill_views_dispatch(lv_ctx* ctx, const RayView* d_rays, const TileQueue& Q,
                                uint32_t ctas, uint32_t checks, cudaStream_t s)
{
    auto k = raycast_refill_views_kernel<DT, F, EDGE>;
    uint32_t grid = resident_ctas(ctx, k, kRefillThreads, 0);
    if (ctas)
    {
        int sms = 152;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        grid = uint32_t(sms) * ctas;
    }
    k<<<grid, kRefillThreads, 0, s>>>(d_rays, Q, checks);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

/* A fixed-pitch kernel decides the brick layout from its pitch at compile
 * time (voxel quads for uint8 rows of kQuadMinRow to kQuadMaxRow); a view
 * whose pool keeps such bricks compact (LV_BRICKS_COMPACT) takes the
 * generic-pitch kernels, which read the layout from the view. */
bool fixed_pitch_layout(const RayView& V)
{
    return V.dtype != LV_DT_UINT8 || (V.quads != 0) == quad_layout(V.dtype, V.N[0]);
}

/* Scratch bytes of the longest-first order of V's tiles. */
size_t order_bytes_of(const RayView& V, const lv_render_launch& L)
{
    const size_t total =
        size_t((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
    return 2 * kTileBuckets * sizeof(uint32_t) + ((total + 15) & ~size_t(15)) +
           sizeof(uint32_t) * total;
}

/* Longest-first order of the tiles of V (a memset and two small launches)
 * in `scratch` (tile_order_bytes); nullptr for raster order. */
const uint32_t* tile_order(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                           uint8_t* scratch, cudaStream_t s, lv_status& st)
{
    st = LV_OK;
    if (L.order != LV_ORDER_LONGEST_FIRST)
        return nullptr;
    const uint32_t tiles_x = (V.W + L.tile_w - 1) / L.tile_w;
    const uint32_t total = tiles_x * ((V.H + L.tile_h - 1) / L.tile_h);
    const size_t hist_bytes = 2 * kTileBuckets * sizeof(uint32_t);
    const size_t key_bytes = (size_t(total) + 15) & ~size_t(15);
    cudaError_t e = cudaMemsetAsync(scratch, 0, hist_bytes, s);
    if (e != cudaSuccess)
    {
        st = cuda_fail(ctx, e, "tile order");
        return nullptr;
    }
    uint32_t* hist = reinterpret_cast<uint32_t*>(scratch);
    uint8_t* keys = scratch + hist_bytes;
    uint32_t* order = reinterpret_cast<uint32_t*>(keys + key_bytes);
    float diag = 0.f;
    for (int a = 0; a < 3; ++a)
        diag += (V.gmax[a] - V.gmin[a]) * (V.gmax[a] - V.gmin[a]);
    const float per_length = float(kTileBuckets) / std::sqrt(diag);
    const uint32_t blocks = (total + 255) / 256;
    tile_key_kernel<<<blocks, 256, 0, s>>>(V, L.tile_w, L.tile_h, tiles_x, total, per_length,
                                           keys, hist);
    tile_order_kernel<<<blocks, 256, 0, s>>>(keys, hist, order, total);
    ctx->kernels += 2u;
    e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        st = cuda_fail(ctx, e, "tile order");
        return nullptr;
    }
    return order;
}

/* lv_render's scratch for the tile order of V. */
uint8_t* render_order_scratch(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                              lv_status& st)
{
    st = LV_OK;
    if (L.order != LV_ORDER_LONGEST_FIRST)
        return nullptr;
    DeviceBuffer& buf = ctx->renderer->tiles;
    const cudaError_t e = buf.reserve(order_bytes_of(V, L));
    if (e != cudaSuccess)
        st = cuda_fail(ctx, e, "tile order");
    return buf.as<uint8_t>();
}

} // namespace

namespace
{
/* Restricts V's rect to the pixels whose ray can reach the volume (its screen
 * rectangle) and gives the others (W = 0: none), so that the ray cast launches
 * no blocks for them (85 % of the pixels of a 1080p orbit frame). Frame times:
 * a float volume at 1001 x 701 477 -> 449 us, the nearest filter at 1024 x 768
 * 406 -> 391, 2048^3 uint8 at 1080p 277 -> 274. */
ClearRect shrink_to_candidates(RayView& V)
{
    /* corners on multiples of 8 pixels: a row of a tile is a whole 128-byte
     * line of the frame */
    uint32_t x0 = std::max(V.x0, V.cull[0] & ~7u), x1 = std::min(V.x0 + V.W, V.cull[2]);
    uint32_t y0 = std::max(V.y0, V.cull[1] & ~7u), y1 = std::min(V.y0 + V.H, V.cull[3]);
    if (x0 >= x1 || y0 >= y1)
    {
        /* nothing to see: one pixel, for the launch to report the frame */
        x0 = V.x0;
        y0 = V.y0;
        x1 = x0 + 1;
        y1 = y0 + 1;
    }
    ClearRect C{V.out, V.FW, V.x0, V.y0, V.W, V.H, x0, y0, x1, y1};
    if (uint64_t(x1 - x0) * (y1 - y0) == uint64_t(V.W) * V.H)
        C.W = 0;
    V.x0 = x0;
    V.y0 = y0;
    V.W = x1 - x0;
    V.H = y1 - y0;
    return C;
}

dim3 clear_grid(const ClearRect& C)
{
    return dim3(std::max(1u, (C.W + 255) / 256), std::min(std::max(C.H, 1u), 1024u));
}
} // namespace

lv_status launch_frame_clear(lv_ctx* ctx, RayView& V, uint64_t cells, cudaStream_t s,
                             cudaEvent_t ready, bool& more)
{
    const ClearRect C = shrink_to_candidates(V);
    /* up to 2 million pixels (5 us) with the rest; more would hold up the
     * residency pass, so they get a launch of their own behind `ready` */
    more = uint64_t(C.W) * C.H > (1u << 21);
    ClearRect now = C;
    if (more)
        now.W = 0;
    /* enough blocks for the larger of the two jobs: a narrow rect of a deep
     * octree has few pixels and many cells */
    const uint32_t for_cells = uint32_t(std::min<uint64_t>((cells + 1023) / 1024, 608u));
    dim3 grid(for_cells);
    if (now.W)
    {
        grid = clear_grid(now);
        grid.y = std::max(grid.y, (for_cells + grid.x - 1) / grid.x);
    }
    frame_clear_kernel<<<grid, 256, 0, s>>>(V.counters, const_cast<uint32_t*>(V.leaf), cells, now);
    LV_CUDA(ctx, cudaGetLastError());
    LV_CUDA(ctx, cudaEventRecord(ready, s));
    if (more)
        clear_outside_kernel<<<clear_grid(C), 256, 0, s>>>(C);
    ctx->kernels += more ? 2u : 1u;
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

uint64_t candidate_rays(const RayView& V)
{
    const uint32_t x0 = std::max(V.x0, V.cull[0]), x1 = std::min(V.x0 + V.W, V.cull[2]);
    const uint32_t y0 = std::max(V.y0, V.cull[1]), y1 = std::min(V.y0 + V.H, V.cull[3]);
    return x0 < x1 && y0 < y1 ? uint64_t(x1 - x0) * (y1 - y0) : 0;
}

namespace
{
/* The fixed pitch whose kernels render V (34, 66, 130: the 32^3, 64^3 and
 * 128^3 bricks with an overlap of 1), or 0. */
uint32_t fixed_pitch(const RayView& V)
{
    const bool fixed = V.edge == 0 && V.filter == LV_FILTER_TRILINEAR && V.N[0] == V.N[1] &&
                       (V.N[0] == 34 || V.N[0] == 66 || V.N[0] == 130) && fixed_pitch_layout(V);
    return fixed ? V.N[0] : 0;
}

/* The default launch. */
bool splittable(const lv_render_launch& L)
{
    return L.kind == LV_LAUNCH_TILE_GRID && L.tile_w == 8 && L.tile_h == 8 && L.lookahead;
}

/* Lanes that share a ray in a launch of `rays` candidate rays (pixels that
 * can reach the volume) under the default launch; other launch shapes keep
 * one lane per ray. Few rays leave most of the 152 SMs' issue slots idle
 * behind chains of dependent loads, so their samples go to more lanes; the
 * exchange costs instructions, which a frame that fills the GPU pays for
 * unless the samples of a ray share cache lines that neighbouring rays do not:
 * the ray's step is well below a pixel (px_per_step), a pixel not below a
 * voxel. Ray-cast us with 1 / 4 / 8 lanes, by rays and (px_per_voxel,
 * px_per_step), orbits at 1.6 volume diagonals:
 *                    13 600               114 000                395 000
 *   uint8 64^3       81  32  25 ( .6, .3) 515  365 395 (1.0, .3)  1012 1020 1225 ( .9,  .5)
 *    LOD 2 px        36  18  18 (1.3, .6) 182  184 213 (2.0, .5)   920 1000 1212 (1.8,  .5)
 *   uint8 32^3       87  38  29 ( .6, .3) 213  171 197 (1.0, .5)   389  447  577 (1.8,  .9)
 *   uint16 64^3      87  36  29 ( .6, .3) 883  532 507 (1.0, .3)  2204 1424 1597 ( .9,  .5)
 *    LOD 3 px        39  20  18 (1.3, .6) 100  112 137 (2.0, 1.)   591  563  732 (1.8,  .9)
 *   uint16 128^3    122  62  43 ( .6, .2) 247  188 195 (2.0, .5)   718  666  774 (1.8,  .9)
 *   float 380^3     571 155  92 ( .2, .1) 548  265 282 ( .7, .3)   992  669  836 (1.2,  .6)
 *   float 128^3      91  34  28 ( .6, .3) 101  105 132 (2.0, 1.)   234  286  394 (3.7, 1.8)
 *   int16 300^3     467 135  84 ( .3, .1) 563  387 391 ( .8, .4)  1263  914 1113 (1.6,  .8)
 *   nearest 512^3   399 111  66 ( .2, .2) 340  212 235 ( .5, .5)   615  537  699 ( .9,  .9)
 *   nearest 128^3   146  50  38 ( .6, .2) 146  158 191 (2.0, .5)   354  448  590 (3.7,  .9)
 *   clamped 256^3   265  74  57 ( .3, .2) 867  318 286 (1.0, .5)  1119  689  781 (1.8,  .9)
 * The trilinear uint8 kernels have the fewest loads per sample, so they fill
 * the issue slots with the fewest rays; clamped taps have the longest chains.
 *
 * uint16: rays * px_per_step separates what gains from what loses. Up to
 * 250 000 four lanes pay (1024^3 in 64^3 bricks: 240 000 rays, .65: 391 / 264
 * us; 373 000, .41: 805 / 623; inside 173 000, .96: 361 / 283), above 500 000
 * they do not (581 000, 1.0: 428 / 502; inside 480 000, 1.6: 526 / 602; in 128^3
 * bricks 581 000, 1.0, 4096 table entries: 479 / 583). Between the two it is the
 * data: long rays through a clear volume gain (512^3, 362 000, .9: 1143 / 946),
 * rays that end early lose (581 000, .5: 1089 / 1179), so the limits by voxel
 * size decide there; bricks below 64^3 lose (256^3 in 32^3, 373 000, .8: 232 /
 * 262; clear 311 / 344). Clamped taps depend on the data throughout (512^3,
 * about 1 M rays: uint16 3682 / 1994 and uint8 in quads 3505 / 1958 through a
 * clear volume, uint8 in quads 982 / 1167 where rays end early), but for voxels
 * stored as one byte, whose taps share most lines: product above 600 000, 380^3
 * uint8 in 48^3 bricks 993 / 1131, 256^3 int8 911 / 1104. The nearest filter's single load gains nothing where
 * the near voxels are magnified (px_near): 512^3 uint16, 494 000 rays, 1.7: 457 /
 * 580, 344 000, 1.45: 356 / 415; but 471 000, 1.3: 870 / 864, 328 000, 1.1: 426 /
 * 374. */
uint32_t split_lanes(const RayView& V, const lv_render_launch& L, uint64_t rays)
{
    if (!splittable(L))
        return 1;
    const float p = std::max(V.px_per_voxel, 0.01f), r = float(rays);
    const float step = std::max(V.px_per_step, 0.001f);
    float eight, four; /* rays up to which that many lanes share a ray */
    if (rays > candidate_rays(V))
    {
        /* views cast together fill each other's gaps: few in all (two small
         * views 217 -> 180 us; three with 200 000 rays 338 -> 357) */
        eight = 8192.f;
        four = 81920.f;
    }
    else if (V.filter != LV_FILTER_TRILINEAR)
    {
        eight = 32768.f;
        four = p < 1.2f ? std::max(std::min(500000.f, 700000.f / (V.px_near * V.px_near)), 90000.f)
                        : 90000.f;
    }
    else if (V.edge)
    {
        eight = 100000.f;
        four = 2000000.f / p;
        if (V.dtype == LV_DT_INT8 || (V.dtype == LV_DT_UINT8 && !V.quads))
            four = std::min(four, 600000.f / step);
    }
    else if (V.dtype == LV_DT_UINT8)
    {
        eight = 16384.f;
        four = p < 1.25f ? 230000.f : 90000.f;
    }
    else
    {
        eight = V.dtype == LV_DT_UINT16 ? 16384.f : 32768.f;
        four = p < 1.4f ? 600000.f : (p < 1.9f ? 800000.f : 500000.f) / p;
        if (V.dtype == LV_DT_UINT16)
            four = std::max(250000.f / step, V.N[0] >= 64u ? std::min(four, 500000.f / step) : 0.f);
    }
    return r <= eight ? 8 : r <= four ? 4 : 1;
}
} // namespace

RayLaunch ray_launch(const RayView& V, const lv_render_launch& L, uint64_t rays, uint32_t forced)
{
    RayLaunch R{L, splittable(L) && forced ? forced : split_lanes(V, L, rays)};
    if (R.lanes > 1)
    {
        /* 64 threads: 4 x 4 pixels of 4 lanes or 4 x 2 of 8 */
        R.shape.tile_w = 4;
        R.shape.tile_h = 16 / R.lanes;
    }
    else if (V.dtype != LV_DT_UINT8 && V.dtype != LV_DT_UINT16)
    {
        R.shape.kind = LV_LAUNCH_TILE_GRID;
        const uint32_t px = L.tile_w * L.tile_h;
        if (px == 0 || px > 256 || px % 32 != 0)
        {
            R.shape.tile_w = 8;
            R.shape.tile_h = 16;
        }
    }
    return R;
}

namespace
{
/* Whether the one-lane tile kernel of V runs with 12 blocks an SM rather than
 * 16 (raycast_tiles_roomy_kernel). uint16 taps are eight scattered loads a
 * sample, so where neighbouring rays share few lines (the finest voxels are
 * small on screen, whatever level is rendered) and the table takes its part of
 * the L1, fewer rays at a time hit it more often; magnified voxels are shared
 * and want the issue slots filled. The line by voxel size on screen rises with
 * the table: 0.65 px at 256 entries, 1.3 at 4096 (fourth root); without a
 * fixed pitch the roomy kernel needs 78 registers and pays up to 0.42 and 0.84
 * px. Ray-cast ms with 16 / 12 blocks by (px_finest):
 *   8192^3 in 128^3 bricks, 1080p, inside, 4096 entries  103.6 /  99.4 ( .16)
 *     the same with 256 entries                           87.5 /  84.8 ( .16)
 *   8192^3 in 128^3, orbit at 1.2, 4096 entries, 1080p     8.0 /   7.5 ( .08)
 *   2048^3 in 64^3, orbit at 1.2, 256 entries, 1080p       6.9 /   6.5 ( .31)
 *   1024^3 in 64^3, orbit at 1.2, 4096 entries, 2160p     11.0 /  10.6 (1.2)
 *   2048^3 in 64^3, inside, 4096 entries, 2160p           31.1 /  32.5 (2.9)
 *   1024^3 in 64^3, inside, 256 entries, 1440p             6.7 /   7.1 (3.8)
 *   3072^3 in 96^3, orbit at 1.2, 4096 entries, 2160p     42.4 /  40.5 ( .41)
 *     inside, LOD 2 px, 256 entries, 1080p                19.3 /  20.0 ( .44)
 * Of 300 views none by this rule is over 3 % behind the better of the two, and
 * 124 are 2 to 8 % ahead of 16 blocks. Bricks below 64^3 look up so often that
 * 16 blocks are better or equal (512^3 in 32^3 bricks 1.54 / 1.67), as for
 * uint8 (2048^3 in 64^3, orbit, 3.6 / 3.9) and the nearest filter. */
bool roomy_l1(const RayView& V)
{
    const float line = fixed_pitch(V) ? 0.1625f : 0.105f;
    return V.N[0] >= 64u && V.px_finest < line * std::sqrt(std::sqrt(V.tf_last + 1.0f));
}

template <int DT, int F, int EDGE>
TileKernel one_lane_kernel(const RayView& V, uint32_t lookahead)
{
    if constexpr (DT == LV_DT_UINT16 && F == LV_FILTER_TRILINEAR && EDGE != 1 && EDGE != 34)
        if (lookahead && roomy_l1(V))
            return raycast_tiles_roomy_kernel<DT, F, EDGE, 1>;
    return lookahead ? raycast_tiles_kernel<DT, F, EDGE, 1> : raycast_tiles_kernel<DT, F, EDGE, 0>;
}

/* The kernels of bricks of 34 x 34, 66 x 66 and 130 x 130 voxels in x and y
 * (the 32^3, 64^3 and 128^3 bricks with an overlap of 1) have the pitches as
 * immediates. */
template <int DT>
TileKernel one_lane_kernel(const RayView& V, uint32_t lookahead)
{
    if (V.filter != LV_FILTER_TRILINEAR)
        return V.edge ? one_lane_kernel<DT, LV_FILTER_NEAREST, 1>(V, lookahead)
                      : one_lane_kernel<DT, LV_FILTER_NEAREST, 0>(V, lookahead);
    switch (fixed_pitch(V))
    {
    case 34: return one_lane_kernel<DT, LV_FILTER_TRILINEAR, 34>(V, lookahead);
    case 66: return one_lane_kernel<DT, LV_FILTER_TRILINEAR, 66>(V, lookahead);
    case 130: return one_lane_kernel<DT, LV_FILTER_TRILINEAR, 130>(V, lookahead);
    default:
        return V.edge ? one_lane_kernel<DT, LV_FILTER_TRILINEAR, 1>(V, lookahead)
                      : one_lane_kernel<DT, LV_FILTER_TRILINEAR, 0>(V, lookahead);
    }
}

/* The kernel of V as launch R with one CTA per tile (null: unknown type). */
TileKernel tile_kernel(const RayView& V, const RayLaunch& R)
{
    if (V.dtype != LV_DT_UINT8 && V.dtype != LV_DT_UINT16)
        return other_type_kernel(V, R);
    if (R.lanes > 1)
        return split_kernel(V, R.lanes, fixed_pitch(V));
    return V.dtype == LV_DT_UINT8 ? one_lane_kernel<LV_DT_UINT8>(V, R.shape.lookahead)
                                  : one_lane_kernel<LV_DT_UINT16>(V, R.shape.lookahead);
}

uint32_t tiles_of(const RayView& V, const lv_render_launch& L)
{
    return ((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
}
} // namespace

lv_status prepare_frame_order(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                              cudaStream_t side, const uint32_t*& order)
{
    order = nullptr;
    const RayLaunch R = ray_launch(V, L, candidate_rays(V), ctx->test_lanes);
    const lv_render_launch& T = R.shape;
    const uint32_t threads = T.tile_w * T.tile_h * R.lanes;
    if (T.kind == LV_LAUNCH_TILE_GRID && threads <= 64)
    {
        /* tiles that are all resident at once start together in any order: no
         * order is computed, three launches fewer. Up to 12 blocks an SM: with
         * more, raster order may leave the long tiles to few SMs (nearest
         * filter, 102 x 744, 14 an SM: 82.4 us a frame ordered, 84.8 not). */
        const TileKernel k = tile_kernel(V, R);
        uint32_t& resident = ctx->renderer->resident_tiles[{k, threads}];
        if (k && resident == 0)
            resident = resident_ctas(ctx, k, int(threads), 0, 12);
        if (tiles_of(V, T) <= resident)
            return LV_OK;
    }
    if (T.kind == LV_LAUNCH_GRID || T.order != LV_ORDER_LONGEST_FIRST)
        return LV_OK;
    lv_status st = LV_OK;
    uint8_t* scratch = render_order_scratch(ctx, V, T, st);
    if (st != LV_OK)
        return st;
    order = tile_order(ctx, V, T, scratch, side, st);
    return st;
}

namespace
{
/* The tile order of a launch (null: raster order): lv_render's (scratch ==
 * nullptr), computed ahead on its side stream, or a batch view's, computed now
 * on `s`. */
const uint32_t* frame_order(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                            uint8_t* scratch, cudaStream_t s, lv_status& st)
{
    st = LV_OK;
    return scratch ? tile_order(ctx, V, L, scratch, s, st) : ctx->renderer->pre_order;
}

template <int DT, int F, int EDGE>
lv_status refill_dispatch(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                          cudaStream_t s)
{
    lv_status st = LV_OK;
    const uint32_t* order = frame_order(ctx, V, L, nullptr, s, st);
    if (st != LV_OK)
        return st;
    auto k = raycast_refill_kernel<DT, F, EDGE>;
    const uint32_t tiles = ((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
    const uint32_t warps = kRefillThreads / 32;
    const uint32_t grid = std::max(1u, std::min(resident_ctas(ctx, k, kRefillThreads, 0),
                                                (tiles + warps - 1) / warps));
    k<<<grid, kRefillThreads, 0, s>>>(V, L.tile_w, L.tile_h, L.samples_per_check, order);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

template <int DT, int F, int EDGE, int LA>
lv_status plain_dispatch_la(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                            cudaStream_t s, uint8_t* scratch)
{
    if (L.kind == LV_LAUNCH_WARP_TILES)
    {
        lv_status st = LV_OK;
        const uint32_t* order = frame_order(ctx, V, L, scratch, s, st);
        if (st != LV_OK)
            return st;
        auto k = raycast_warp_tiles_kernel<DT, F, EDGE, LA>;
        const uint32_t tiles =
            ((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
        const uint32_t grid =
            std::max(1u, std::min(resident_ctas(ctx, k, 128, 0), (tiles + 3) / 4));
        k<<<grid, 128, 0, s>>>(V, L.tile_w, L.tile_h, order);
        LV_CUDA(ctx, cudaGetLastError());
        return LV_OK;
    }
    if (L.kind == LV_LAUNCH_TILE_QUEUE)
    {
        lv_status st = LV_OK;
        const uint32_t* order = frame_order(ctx, V, L, scratch, s, st);
        if (st != LV_OK)
            return st;
        auto k = raycast_queue_kernel<DT, F, EDGE, LA>;
        const uint32_t threads = L.tile_w * L.tile_h;
        const uint32_t tiles =
            ((V.W + L.tile_w - 1) / L.tile_w) * ((V.H + L.tile_h - 1) / L.tile_h);
        const uint32_t grid =
            std::max(1u, std::min(resident_ctas(ctx, k, int(threads), 0), tiles));
        k<<<grid, threads, 0, s>>>(V, L.tile_w, L.tile_h, order);
        LV_CUDA(ctx, cudaGetLastError());
        return LV_OK;
    }
    const dim3 block(L.tile_w, L.tile_h);
    const dim3 grid((V.W + block.x - 1) / block.x, (V.H + block.y - 1) / block.y);
    raycast_kernel<DT, F, EDGE, LA><<<grid, block, 0, s>>>(V);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

template <int DT, int F, int EDGE>
lv_status plain_dispatch(lv_ctx* ctx, const RayView& V, const lv_render_launch& L,
                         cudaStream_t s, uint8_t* scratch)
{
    if (L.kind == LV_LAUNCH_WARP_REFILL)
        return refill_dispatch<DT, F, EDGE>(ctx, V, L, s);
    if (L.lookahead)
        return plain_dispatch_la<DT, F, EDGE, 1>(ctx, V, L, s, scratch);
    return plain_dispatch_la<DT, F, EDGE, 0>(ctx, V, L, s, scratch);
}

/* combination index (batch_group): 0..7 dtype (u8 0 / u16 1), filter,
 * edge; 8..13 trilinear bricks of pitch 34 / 66 / 130 (u8, then u16) */
template <int TFS>
lv_status persistent_by_index(int idx, lv_ctx* ctx, const RayView* d, const TileQueue& Q,
                              uint32_t ctas, size_t smem, cudaStream_t s)
{
    switch (idx)
    {
    case 8: return persistent_dispatch<LV_DT_UINT8, 1, TFS, 34>(ctx, d, Q, ctas, smem, s);
    case 9: return persistent_dispatch<LV_DT_UINT8, 1, TFS, 66>(ctx, d, Q, ctas, smem, s);
    case 10: return persistent_dispatch<LV_DT_UINT8, 1, TFS, 130>(ctx, d, Q, ctas, smem, s);
    case 11: return persistent_dispatch<LV_DT_UINT16, 1, TFS, 34>(ctx, d, Q, ctas, smem, s);
    case 12: return persistent_dispatch<LV_DT_UINT16, 1, TFS, 66>(ctx, d, Q, ctas, smem, s);
    case 13: return persistent_dispatch<LV_DT_UINT16, 1, TFS, 130>(ctx, d, Q, ctas, smem, s);
    case 0: return persistent_dispatch<LV_DT_UINT8, 0, TFS, 0>(ctx, d, Q, ctas, smem, s);
    case 1: return persistent_dispatch<LV_DT_UINT8, 0, TFS, 1>(ctx, d, Q, ctas, smem, s);
    case 2: return persistent_dispatch<LV_DT_UINT8, 1, TFS, 0>(ctx, d, Q, ctas, smem, s);
    case 3: return persistent_dispatch<LV_DT_UINT8, 1, TFS, 1>(ctx, d, Q, ctas, smem, s);
    case 4: return persistent_dispatch<LV_DT_UINT16, 0, TFS, 0>(ctx, d, Q, ctas, smem, s);
    case 5: return persistent_dispatch<LV_DT_UINT16, 0, TFS, 1>(ctx, d, Q, ctas, smem, s);
    case 6: return persistent_dispatch<LV_DT_UINT16, 1, TFS, 0>(ctx, d, Q, ctas, smem, s);
    default: return persistent_dispatch<LV_DT_UINT16, 1, TFS, 1>(ctx, d, Q, ctas, smem, s);
    }
}

lv_status refill_views_by_index(int idx, lv_ctx* ctx, const RayView* d, const TileQueue& Q,
                                uint32_t ctas, uint32_t checks, cudaStream_t s)
{
    /* the fixed-pitch groups take the general trilinear kernels */
    if (idx >= 8 && idx <= 10)
        idx = 2;
    else if (idx >= 11 && idx <= 13)
        idx = 6;
    switch (idx)
    {
    case 0: return refill_views_dispatch<LV_DT_UINT8, 0, 0>(ctx, d, Q, ctas, checks, s);
    case 1: return refill_views_dispatch<LV_DT_UINT8, 0, 1>(ctx, d, Q, ctas, checks, s);
    case 2: return refill_views_dispatch<LV_DT_UINT8, 1, 0>(ctx, d, Q, ctas, checks, s);
    case 3: return refill_views_dispatch<LV_DT_UINT8, 1, 1>(ctx, d, Q, ctas, checks, s);
    case 4: return refill_views_dispatch<LV_DT_UINT16, 0, 0>(ctx, d, Q, ctas, checks, s);
    case 5: return refill_views_dispatch<LV_DT_UINT16, 0, 1>(ctx, d, Q, ctas, checks, s);
    case 6: return refill_views_dispatch<LV_DT_UINT16, 1, 0>(ctx, d, Q, ctas, checks, s);
    default: return refill_views_dispatch<LV_DT_UINT16, 1, 1>(ctx, d, Q, ctas, checks, s);
    }
}
} // namespace

size_t tile_order_bytes(const RayView& V, const RayLaunch& R)
{
    return order_bytes_of(V, R.shape);
}

int batch_group(const RayView& V)
{
    const int v = kernel_variant(V.dtype, V.filter, V.edge);
    const uint32_t pitch = fixed_pitch(V);
    if (v >= 8 || pitch == 0)
        return v < 8 ? v : kBatchGroups + v;
    return 8 + (V.dtype == LV_DT_UINT16 ? 3 : 0) + (pitch == 34 ? 0 : pitch == 66 ? 1 : 2);
}

/* 0..7: uint8 / uint16 x filter x edge; 8..11: the other voxel types x
 * filter x edge */
int kernel_variant(uint32_t dtype, uint32_t filter, uint32_t edge)
{
    const int fe = (filter == LV_FILTER_TRILINEAR ? 2 : 0) + (edge ? 1 : 0);
    if (dtype != LV_DT_UINT8 && dtype != LV_DT_UINT16)
        return 8 + fe;
    return (dtype == LV_DT_UINT16 ? 4 : 0) + fe;
}

lv_status launch_raycast(lv_ctx* ctx, const RayView& V, cudaStream_t s)
{
    if (V.dtype > LV_DT_INT32)
        return fail(ctx, LV_EINVAL, "unknown voxel type");
    /* the ray-cast kernels derive the samples per ray themselves */
    const RayLaunch R = ray_launch(V, ctx->launch, candidate_rays(V), ctx->test_lanes);
    ctx->renderer->lanes = R.lanes;
    return launch_view_raycast(ctx, V, R, nullptr, s);
}

lv_status launch_view_raycast(lv_ctx* ctx, const RayView& V, const RayLaunch& R,
                              uint8_t* order_scratch, cudaStream_t s)
{
    const lv_render_launch& L = R.shape;
    ++ctx->kernels; /* whichever launch it is */
    if (L.kind == LV_LAUNCH_TILE_GRID)
    {
        lv_status st = LV_OK;
        const uint32_t* order = frame_order(ctx, V, L, order_scratch, s, st);
        if (st != LV_OK)
            return st;
        const TileKernel k = tile_kernel(V, R);
        if (!k)
            return fail(ctx, LV_EINVAL, "unknown voxel type");
        k<<<tiles_of(V, L), L.tile_w * L.tile_h * R.lanes, 0, s>>>(V, L.tile_w, L.tile_h, order);
        LV_CUDA(ctx, cudaGetLastError());
        return LV_OK;
    }
    switch (kernel_variant(V.dtype, V.filter, V.edge))
    {
    case 0: return plain_dispatch<LV_DT_UINT8, 0, 0>(ctx, V, L, s, order_scratch);
    case 1: return plain_dispatch<LV_DT_UINT8, 0, 1>(ctx, V, L, s, order_scratch);
    case 2: return plain_dispatch<LV_DT_UINT8, 1, 0>(ctx, V, L, s, order_scratch);
    case 3: return plain_dispatch<LV_DT_UINT8, 1, 1>(ctx, V, L, s, order_scratch);
    case 4: return plain_dispatch<LV_DT_UINT16, 0, 0>(ctx, V, L, s, order_scratch);
    case 5: return plain_dispatch<LV_DT_UINT16, 0, 1>(ctx, V, L, s, order_scratch);
    case 6: return plain_dispatch<LV_DT_UINT16, 1, 0>(ctx, V, L, s, order_scratch);
    default: return plain_dispatch<LV_DT_UINT16, 1, 1>(ctx, V, L, s, order_scratch);
    }
}

lv_status launch_views_pipeline(lv_ctx* ctx, const ResolveView* d_resolve,
                                const RayView* d_rays, uint32_t n, cudaStream_t s)
{
    resolve_views_kernel<<<dim3(8, n), 256, 0, s>>>(d_resolve);
    prune_views_kernel<<<dim3(8, n), 256, 0, s>>>(d_resolve);
    leaf_fill_views_kernel<<<dim3(16, n), 256, 0, s>>>(d_resolve);
    step_views_kernel<<<(n + 127) / 128, 128, 0, s>>>(d_rays, n);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

lv_status launch_batch_order(lv_ctx* ctx, const RayView* d_rays, const TileQueue& Q,
                             uint32_t max_items, uint8_t* keys, uint32_t* hist,
                             uint32_t* order, cudaStream_t s)
{
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const uint32_t blocks =
        std::max(1u, std::min((max_items + 255) / 256, uint32_t(sms) * 4u));
    LV_CUDA(ctx, cudaMemsetAsync(hist, 0, 2 * kTileBuckets * sizeof(uint32_t), s));
    batch_key_kernel<<<blocks, 256, 0, s>>>(d_rays, Q, keys, hist);
    batch_order_kernel<<<blocks, 256, 0, s>>>(Q, keys, hist, order);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}

lv_status launch_persistent(lv_ctx* ctx, int variant, const lv_batch_config& cfg,
                            const RayView* d_rays, const TileQueue& Q, uint32_t tfn_max,
                            cudaStream_t s)
{
    if (cfg.queue == LV_QUEUE_WARP_REFILL)
        return refill_views_by_index(variant, ctx, d_rays, Q, cfg.ctas_per_sm,
                                     cfg.samples_per_check, s);
    const size_t smem = cfg.tf_shared ? size_t(tfn_max) * 2 * sizeof(float4) : 0;
    if (cfg.tf_shared)
        return persistent_by_index<1>(variant, ctx, d_rays, Q, cfg.ctas_per_sm, smem, s);
    return persistent_by_index<0>(variant, ctx, d_rays, Q, cfg.ctas_per_sm, smem, s);
}

} // namespace lv

extern "C" lv_status lv_frame_to_rgba8(lv_ctx* ctx, const float* d_rgba,
                                       uint32_t width, uint32_t height,
                                       uint8_t* d_out, void* stream)
{
    using namespace lv;
    if (!ctx || (!d_rgba && width * height) || (!d_out && width * height))
        return fail(ctx, LV_EINVAL, "null argument");
    const uint64_t n = uint64_t(width) * height;
    if (n == 0)
        return LV_OK;
    LV_CUDA(ctx, cudaSetDevice(ctx->device));
    const uint32_t blocks = uint32_t(std::min<uint64_t>((n + 255) / 256, 4096));
    to_rgba8_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4*>(d_rgba), reinterpret_cast<uchar4*>(d_out), n);
    LV_CUDA(ctx, cudaGetLastError());
    return LV_OK;
}
