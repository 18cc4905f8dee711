/*
 * Procedural fBm volume: fractal Brownian motion over improved Perlin noise
 * (K. Perlin, "Improving Noise", SIGGRAPH 2002: quintic fade, 12 edge
 * gradients picked by the low 4 bits of the hash, a 256-entry permutation
 * table repeated twice), `octaves` octaves of lacunarity and gain, mapped
 * linearly from [-1, 1] to the full range of the voxel type.
 *
 * The permutation is the identity shuffled by Fisher-Yates with SplitMix64
 * draws from the seed (j = draw mod (i + 1), i from 255 down to 1). A voxel
 * at level-L coordinate g (clamped to the level's extent, as the blob
 * volumes) samples the field at x = (g + 0.5) * 2^(depth-1-L) * frequency /
 * max(voxels), in finest-level voxel units scaled so that `frequency` noise
 * periods span the volume.
 *
 * Every float operation is IEEE single precision in a fixed order with no
 * contraction (the device code uses explicit round-to-nearest intrinsics,
 * the host code is built without FP contraction), so the host generator,
 * which a data-source plugin calls per brick, and the device generator,
 * which writes bricks straight into the pool, give the same bytes.
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>

#include "lv_runtime.h"

namespace lv
{
namespace
{
inline uint64_t splitmix_draw(uint64_t& s)
{
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

/* Operations shared by the host and device generators: FADD/FMUL with
 * round-to-nearest and no fusion. */
struct HostOps
{
    static float add(float a, float b) { return a + b; }
    static float sub(float a, float b) { return a - b; }
    static float mul(float a, float b) { return a * b; }
};
struct DeviceOps
{
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
};

template <typename O>
__host__ __device__ __forceinline__ float fade(float t)
{
    /* t^3 (t (6 t - 15) + 10) */
    const float a = O::add(O::mul(t, O::sub(O::mul(t, 6.0f), 15.0f)), 10.0f);
    return O::mul(O::mul(O::mul(t, t), t), a);
}

template <typename O>
__host__ __device__ __forceinline__ float lerp(float t, float a, float b)
{
    return O::add(a, O::mul(t, O::sub(b, a)));
}

template <typename O>
__host__ __device__ __forceinline__ float grad(uint32_t h, float x, float y, float z)
{
    h &= 15u;
    const float u = h < 8u ? x : y;
    const float v = h < 4u ? y : (h == 12u || h == 14u ? x : z);
    return O::add((h & 1u) ? -u : u, (h & 2u) ? -v : v);
}

template <typename O>
__host__ __device__ __forceinline__ float noise3(const uint16_t* P, float x, float y, float z)
{
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const uint32_t X = uint32_t(int32_t(fx)) & 255u, Y = uint32_t(int32_t(fy)) & 255u,
                   Z = uint32_t(int32_t(fz)) & 255u;
    x = O::sub(x, fx);
    y = O::sub(y, fy);
    z = O::sub(z, fz);
    const float u = fade<O>(x), v = fade<O>(y), w = fade<O>(z);
    const uint32_t A = P[X] + Y, AA = P[A] + Z, AB = P[A + 1] + Z;
    const uint32_t B = P[X + 1] + Y, BA = P[B] + Z, BB = P[B + 1] + Z;
    const float x1 = O::sub(x, 1.0f), y1 = O::sub(y, 1.0f), z1 = O::sub(z, 1.0f);
    const float l00 = lerp<O>(u, grad<O>(P[AA], x, y, z), grad<O>(P[BA], x1, y, z));
    const float l10 = lerp<O>(u, grad<O>(P[AB], x, y1, z), grad<O>(P[BB], x1, y1, z));
    const float l01 = lerp<O>(u, grad<O>(P[AA + 1], x, y, z1), grad<O>(P[BA + 1], x1, y, z1));
    const float l11 = lerp<O>(u, grad<O>(P[AB + 1], x, y1, z1), grad<O>(P[BB + 1], x1, y1, z1));
    return lerp<O>(w, lerp<O>(v, l00, l10), lerp<O>(v, l01, l11));
}

template <typename O>
__host__ __device__ __forceinline__ float fbm(const uint16_t* P, const lv_fbm_params& f, float x,
                                              float y, float z)
{
    float sum = 0.0f, amp = 1.0f, freq = 1.0f;
    for (uint32_t o = 0; o < f.octaves; ++o)
    {
        sum = O::add(sum, O::mul(amp, noise3<O>(P, O::mul(x, freq), O::mul(y, freq),
                                                O::mul(z, freq))));
        amp = O::mul(amp, f.gain);
        freq = O::mul(freq, f.lacunarity);
    }
    return sum;
}

/* [-1, 1] -> [0, full scale], rounded half up */
template <typename O>
__host__ __device__ __forceinline__ uint32_t quantise(float v, float full)
{
    v = fminf(fmaxf(v, -1.0f), 1.0f);
    const float q = O::add(O::mul(O::mul(O::add(v, 1.0f), 0.5f), full), 0.5f);
    return uint32_t(floorf(q));
}

/* Per-brick sampling constants. */
struct FbmBrick
{
    int32_t base[3];   /* level coordinate of the brick's first voxel */
    int32_t last[3];   /* level extent - 1 */
    uint32_t N[3];
    float scale;       /* 2^(depth-1-L) * frequency / max(voxels) */
};

__host__ __device__ __forceinline__ FbmBrick brick_consts(const lv_volume_info& v,
                                                          const lv_fbm_params& f, uint64_t id)
{
    FbmBrick b;
    const uint32_t L = nid_level(id);
    const uint32_t shift = v.depth - 1u - L;
    const uint32_t s = 1u << shift;
    const uint32_t pos[3] = {nid_x(id), nid_y(id), nid_z(id)};
    uint32_t vmax = v.voxels[0];
    vmax = vmax > v.voxels[1] ? vmax : v.voxels[1];
    vmax = vmax > v.voxels[2] ? vmax : v.voxels[2];
    for (int a = 0; a < 3; ++a)
    {
        b.N[a] = v.max_block[a];
        const uint32_t B = v.max_block[a] - 2u * v.overlap[a];
        b.base[a] = int32_t(pos[a] * B) - int32_t(v.overlap[a]);
        b.last[a] = int32_t((v.voxels[a] + s - 1u) >> shift) - 1;
    }
    b.scale = float(s) * (f.frequency / float(vmax));
    return b;
}

template <typename O>
__host__ __device__ __forceinline__ float fbm_at(const uint16_t* P, const lv_fbm_params& f,
                                                 const FbmBrick& b, uint32_t i, uint32_t j,
                                                 uint32_t k)
{
    auto clampi = [](int32_t g, int32_t hi) { return g < 0 ? 0 : (g > hi ? hi : g); };
    const int32_t gi = clampi(b.base[0] + int32_t(i), b.last[0]);
    const int32_t gj = clampi(b.base[1] + int32_t(j), b.last[1]);
    const int32_t gk = clampi(b.base[2] + int32_t(k), b.last[2]);
    const float x = O::mul(O::add(float(gi), 0.5f), b.scale);
    const float y = O::mul(O::add(float(gj), 0.5f), b.scale);
    const float z = O::mul(O::add(float(gk), 0.5f), b.scale);
    return fbm<O>(P, f, x, y, z);
}

/* Coefficients in {-1, 0, 1} of a corner gradient: grad(h, x, y, z) is the
 * sum of the two of sx * x, sy * y, sz * z that are not 0 (grad<O>'s choice
 * of h & 15). */
__device__ __forceinline__ float4 gradient(uint32_t h)
{
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float su = (h & 1u) ? -1.0f : 1.0f, sv = (h & 2u) ? -1.0f : 1.0f;
    if (h < 8u)
        g.x = su;
    else
        g.y = su;
    if (h < 4u)
        g.y = sv;
    else if (h == 12u || h == 14u)
        g.x = sv;
    else
        g.z = sv;
    return g;
}

/* Packed pairs: each half rounds as the scalar operation (a - b as
 * fma(b, -1, a), one rounding). A packed product followed by a packed sum is
 * compiled into one fused operation even where both carry .rn (measured), so
 * the product is itself a fused one, with a -0 that the compiler cannot
 * know: a * b + -0 is a * b rounded, and nothing is left to fuse. */
__constant__ float2 kMinusZero = {-0.0f, -0.0f};
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    return __ffma2_rn(a, b, kMinusZero);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    return __ffma2_rn(b, both(-1.0f), a);
}
__device__ __forceinline__ float2 lerp2(float2 t, float2 a, float2 b)
{
    return __fadd2_rn(a, mul2(t, sub2(b, a)));
}
__device__ __forceinline__ float2 fade2(float2 t)
{
    const float2 a = __fadd2_rn(
        mul2(t, __fadd2_rn(mul2(t, both(6.0f)), both(-15.0f))), both(10.0f));
    return mul2(mul2(mul2(t, t), t), a);
}

/* The gradients at a lattice edge's two ends in z, as functions of x: the
 * value is sx * x + c. sx is 0 or +-1 and c holds the y and z terms (one of
 * them when sx is not 0), so every product is exact and fma(sx, x, c) is
 * grad<O>'s one rounding. */
struct EdgeGrad
{
    float2 sx, c;
};

__device__ __forceinline__ EdgeGrad edge_grad(const float4& lo, const float4& hi, float y,
                                              float2 z)
{
    EdgeGrad e;
    e.sx = make_float2(lo.x, hi.x);
    e.c = __ffma2_rn(make_float2(lo.y, hi.y), both(y), mul2(make_float2(lo.z, hi.z), z));
    return e;
}

/* One brick per blockIdx.y; each thread takes runs of R consecutive voxels
 * of a row (x), strided over blockIdx.x and the threads. Along a run only x
 * changes, so per octave the y and z lattice cells, fractions and fades are
 * computed once, and the eight corner hashes and the y / z parts of their
 * gradients only when the x cell changes; every voxel still gets the values
 * of fbm_at's operations (same roundings, same order; zeros may differ in
 * sign, which no byte shows), so the bytes equal the host generator's.
 *
 * Bound by issue slots, so the arithmetic is in packed pairs: the two ends
 * of each lattice edge in z (corner values, the x and y interpolations) and
 * two voxels of the run (fractions, fades, the octave sum); a corner value
 * is one fused operation on the coefficients of a 16-entry table instead of
 * a selected sum. 130^3 uint16 voxels, 6 octaves: 52 -> 31 us per brick, 57.5
 * -> 27.1 M warp instructions (a packed operation takes the FMA pipe two
 * cycles, so that pipe is 63 % busy, issue 69 %). Runs of 4 or 16 voxels and
 * register bounds for more resident blocks measured 3 to 24 % slower. */
template <int R>
__global__ void __launch_bounds__(256)
    fbm_brick_kernel(lv_volume_info info, lv_fbm_params f, const uint16_t* __restrict__ perm,
                     const uint64_t* __restrict__ ids, const uint64_t* __restrict__ offsets,
                     uint8_t* __restrict__ out, uint64_t brick_bytes)
{
    using O = DeviceOps;
    static_assert(R % 4 == 0, "runs of whole 32-bit words");
    __shared__ uint16_t P[512];
    __shared__ float4 G[16];
    for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x)
        P[i] = perm[i];
    if (threadIdx.x < 16)
        G[threadIdx.x] = gradient(threadIdx.x);
    __syncthreads();
    const uint64_t id = ids[blockIdx.y];
    const FbmBrick b = brick_consts(info, f, id);
    uint8_t* dst = out + (offsets ? offsets[blockIdx.y] : uint64_t(blockIdx.y) * brick_bytes);
    const uint32_t runs_x = (b.N[0] + R - 1) / R;
    const uint32_t n_runs = runs_x * b.N[1] * b.N[2];
    const bool u16 = info.dtype == LV_DT_UINT16;
    const float full = u16 ? 65535.0f : 255.0f;
    auto clampi = [](int32_t g, int32_t hi) { return g < 0 ? 0 : (g > hi ? hi : g); };
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < n_runs;
         w += gridDim.x * blockDim.x)
    {
        /* neighbouring lanes take the same x run of neighbouring rows, so a
         * warp's lanes change x cell at the same voxel (no divergence) */
        const uint32_t j = w % b.N[1], rx = (w / b.N[1]) % runs_x, k = w / (runs_x * b.N[1]);
        const uint32_t i0 = rx * R;
        const uint32_t cnt = min(uint32_t(R), b.N[0] - i0); /* voxels stored */
        const int32_t gj = clampi(b.base[1] + int32_t(j), b.last[1]);
        const int32_t gk = clampi(b.base[2] + int32_t(k), b.last[2]);
        const float y = O::mul(O::add(float(gj), 0.5f), b.scale);
        const float z = O::mul(O::add(float(gk), 0.5f), b.scale);
        float2 xs[R / 2], sum[R / 2];
#pragma unroll
        for (int r = 0; r < R / 2; ++r)
        {
            const int32_t ga = clampi(b.base[0] + int32_t(i0 + 2 * r), b.last[0]);
            const int32_t gb = clampi(b.base[0] + int32_t(i0 + 2 * r + 1), b.last[0]);
            xs[r] = mul2(__fadd2_rn(make_float2(float(ga), float(gb)), both(0.5f)),
                               both(b.scale));
            sum[r] = both(0.0f);
        }
        float amp = 1.0f, freq = 1.0f;
        for (uint32_t o = 0; o < f.octaves; ++o)
        {
            const float yv = O::mul(y, freq), zv = O::mul(z, freq);
            const float fy = floorf(yv), fz = floorf(zv);
            const uint32_t Y = uint32_t(int32_t(fy)) & 255u, Z = uint32_t(int32_t(fz)) & 255u;
            const float yf = O::sub(yv, fy), zf = O::sub(zv, fz);
            const float wz = fade<O>(zf);
            const float2 v = both(fade<O>(yf));
            const float y1 = O::sub(yf, 1.0f);
            const float2 z2 = make_float2(zf, O::sub(zf, 1.0f));
            float cell = __int_as_float(0x7FFFFFFF); /* no cell: differs from all */
            /* edges (dx, dy) from z to z + 1 */
            EdgeGrad e00, e10, e01, e11;
#pragma unroll
            for (int r = 0; r < R / 2; ++r)
            {
                const float2 xv = mul2(xs[r], both(freq));
                const float2 fx = make_float2(floorf(xv.x), floorf(xv.y));
                const float2 xf = sub2(xv, fx);
                const float2 u = fade2(xf);
                const float2 x1 = __fadd2_rn(xf, both(-1.0f));
                float2 n;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const float fxh = h ? fx.y : fx.x;
                    if (fxh != cell)
                    {
                        cell = fxh;
                        const uint32_t X = uint32_t(int32_t(fxh)) & 255u;
                        const uint32_t A = P[X] + Y, AA = P[A] + Z, AB = P[A + 1] + Z;
                        const uint32_t B = P[X + 1] + Y, BA = P[B] + Z, BB = P[B + 1] + Z;
                        e00 = edge_grad(G[P[AA] & 15u], G[P[AA + 1] & 15u], yf, z2);
                        e10 = edge_grad(G[P[BA] & 15u], G[P[BA + 1] & 15u], yf, z2);
                        e01 = edge_grad(G[P[AB] & 15u], G[P[AB + 1] & 15u], y1, z2);
                        e11 = edge_grad(G[P[BB] & 15u], G[P[BB + 1] & 15u], y1, z2);
                    }
                    const float2 xa = both(h ? xf.y : xf.x), xb = both(h ? x1.y : x1.x);
                    const float2 ux = both(h ? u.y : u.x);
                    const float2 l0 = lerp2(ux, __ffma2_rn(e00.sx, xa, e00.c),
                                            __ffma2_rn(e10.sx, xb, e10.c));
                    const float2 l1 = lerp2(ux, __ffma2_rn(e01.sx, xa, e01.c),
                                            __ffma2_rn(e11.sx, xb, e11.c));
                    const float2 m = lerp2(v, l0, l1);
                    (h ? n.y : n.x) = lerp<O>(wz, m.x, m.y);
                }
                sum[r] = __fadd2_rn(sum[r], mul2(both(amp), n));
            }
            amp = O::mul(amp, f.gain);
            freq = O::mul(freq, f.lacunarity);
        }
        const uint64_t row = (uint64_t(k) * b.N[1] + j) * b.N[0] + i0;
        uint32_t q[R];
#pragma unroll
        for (int r = 0; r < R / 2; ++r)
        {
            q[2 * r] = quantise<O>(sum[r].x, full);
            q[2 * r + 1] = quantise<O>(sum[r].y, full);
        }
        /* the lanes' rows are apart, so every store is its own transaction:
         * 32-bit words where the row is aligned for them */
        uint8_t* p = dst + (u16 ? 2u : 1u) * row;
        if (cnt == uint32_t(R) && (uintptr_t(p) & 3u) == 0u)
        {
            if (u16)
            {
#pragma unroll
                for (int r = 0; r < R; r += 2)
                    reinterpret_cast<uint32_t*>(p)[r / 2] = q[r] | (q[r + 1] << 16);
            }
            else
            {
#pragma unroll
                for (int r = 0; r < R; r += 4)
                    reinterpret_cast<uint32_t*>(p)[r / 4] =
                        q[r] | (q[r + 1] << 8) | (q[r + 2] << 16) | (q[r + 3] << 24);
            }
            continue;
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (uint32_t(r) < cnt)
            {
                if (u16)
                    reinterpret_cast<uint16_t*>(p)[r] = uint16_t(q[r]);
                else
                    p[r] = uint8_t(q[r]);
            }
    }
}

bool valid_params(const lv_fbm_params& f)
{
    return f.octaves >= 1 && f.octaves <= 16 && f.frequency > 0.0f &&
           std::isfinite(f.frequency) && std::isfinite(f.gain) && std::isfinite(f.lacunarity);
}

/* Host generation of one brick over `threads` threads (z slabs). */
void fbm_brick_host(const lv_volume_info& info, const lv_fbm_params& f, const uint16_t* P,
                    uint64_t id, void* dst, uint32_t threads)
{
    const FbmBrick b = brick_consts(info, f, id);
    const bool u16 = info.dtype == LV_DT_UINT16;
    const float full = u16 ? 65535.0f : 255.0f;
    auto slab = [&](uint32_t k0, uint32_t k1) {
        for (uint32_t k = k0; k < k1; ++k)
            for (uint32_t j = 0; j < b.N[1]; ++j)
                for (uint32_t i = 0; i < b.N[0]; ++i)
                {
                    const uint32_t q = quantise<HostOps>(fbm_at<HostOps>(P, f, b, i, j, k), full);
                    const size_t idx = (size_t(k) * b.N[1] + j) * b.N[0] + i;
                    if (u16)
                        static_cast<uint16_t*>(dst)[idx] = uint16_t(q);
                    else
                        static_cast<uint8_t*>(dst)[idx] = uint8_t(q);
                }
    };
    threads = std::max(1u, std::min(threads, b.N[2]));
    if (threads == 1)
    {
        slab(0, b.N[2]);
        return;
    }
    std::vector<std::thread> pool;
    const uint32_t per = (b.N[2] + threads - 1) / threads;
    for (uint32_t t = 1; t < threads; ++t)
    {
        const uint32_t k0 = std::min(b.N[2], t * per), k1 = std::min(b.N[2], k0 + per);
        if (k0 < k1)
            pool.emplace_back(slab, k0, k1);
    }
    slab(0, std::min(b.N[2], per));
    for (auto& th : pool)
        th.join();
}

/* Host data source of an fBm volume (the LV_FBM_HOST placement). */
struct FbmSource
{
    lv_volume_info info;
    lv_fbm_params params;
    std::vector<uint16_t> perm;
    uint32_t threads;
};

int fbm_source_get(void* user, uint64_t id, void* dst, size_t bytes)
{
    const FbmSource* src = static_cast<const FbmSource*>(user);
    const lv_volume_info& v = src->info;
    if (nid_level(id) >= v.depth)
        return 1;
    const uint64_t need = uint64_t(v.max_block[0]) * v.max_block[1] * v.max_block[2] *
                          (v.dtype == LV_DT_UINT16 ? 2u : 1u);
    if (bytes < need)
        return 1;
    fbm_brick_host(v, src->params, src->perm.data(), id, dst, src->threads);
    return 0;
}

void fbm_source_free(void* user) { delete static_cast<FbmSource*>(user); }
} // namespace

std::vector<uint16_t> fbm_permutation(uint64_t seed)
{
    std::vector<uint16_t> p(512);
    for (uint32_t i = 0; i < 256; ++i)
        p[i] = uint16_t(i);
    uint64_t s = seed;
    for (uint32_t i = 255; i >= 1; --i)
    {
        const uint32_t j = uint32_t(splitmix_draw(s) % (i + 1u));
        std::swap(p[i], p[j]);
    }
    for (uint32_t i = 0; i < 256; ++i)
        p[256 + i] = p[i];
    return p;
}

lv_status launch_fbm_bricks(lv_ctx* ctx, const lv_volume_info& info, const lv_fbm_params& f,
                            const uint16_t* d_perm, const uint64_t* d_ids, uint32_t n,
                            uint8_t* out, const uint64_t* d_offsets, uint64_t brick_bytes,
                            cudaStream_t s)
{
    for (uint32_t first = 0; first < n; first += kFbmLaunchBricks)
    {
        const uint32_t cnt = std::min(kFbmLaunchBricks, n - first);
        constexpr int R = 8;
        const uint32_t runs =
            (info.max_block[0] + R - 1) / R * info.max_block[1] * info.max_block[2];
        const dim3 grid(std::min(64u, (runs + 255u) / 256u), cnt);
        fbm_brick_kernel<R><<<grid, 256, 0, s>>>(info, f, d_perm, d_ids + first,
                                               d_offsets ? d_offsets + first : nullptr,
                                               d_offsets ? out : out + first * brick_bytes,
                                               brick_bytes);
        LV_CUDA(ctx, cudaGetLastError());
    }
    return LV_OK;
}

} // namespace lv

using namespace lv;

extern "C" lv_status lv_fbm_brick(const lv_volume_info* info, const lv_fbm_params* params,
                                  uint64_t node_id, void* dst, uint32_t n_threads)
{
    if (!info || !params || !dst || !valid_params(*params) || info->depth == 0 ||
        nid_level(node_id) >= info->depth ||
        (info->dtype != LV_DT_UINT8 && info->dtype != LV_DT_UINT16))
        return LV_EINVAL;
    const std::vector<uint16_t> P = fbm_permutation(params->seed);
    fbm_brick_host(*info, *params, P.data(), node_id, dst, n_threads ? n_threads : 1u);
    return LV_OK;
}

extern "C" lv_status lv_fbm_generate(lv_ctx* ctx, const lv_volume_info* info,
                                     const lv_fbm_params* params, const uint64_t* ids,
                                     uint32_t n, void* d_out, void* stream)
{
    if (!ctx || !info || !params || (n && (!ids || !d_out)) || !valid_params(*params) ||
        (info->dtype != LV_DT_UINT8 && info->dtype != LV_DT_UINT16))
        return fail(ctx, LV_EINVAL, "invalid fBm generation arguments");
    for (uint32_t i = 0; i < n; ++i)
        if (nid_level(ids[i]) >= info->depth)
            return fail(ctx, LV_EINVAL, "node id outside the volume");
    if (n == 0)
        return LV_OK;
    std::lock_guard<std::mutex> lock(ctx->mutex);
    LV_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const std::vector<uint16_t> P = fbm_permutation(params->seed);
    DeviceBuffer dperm, dids;
    LV_CUDA(ctx, dperm.reserve(sizeof(uint16_t) * P.size()));
    LV_CUDA(ctx, dids.reserve(sizeof(uint64_t) * n));
    LV_CUDA(ctx, cudaMemcpyAsync(dperm.ptr, P.data(), sizeof(uint16_t) * P.size(),
                                 cudaMemcpyHostToDevice, s));
    LV_CUDA(ctx, cudaMemcpyAsync(dids.ptr, ids, sizeof(uint64_t) * n, cudaMemcpyHostToDevice, s));
    const uint64_t brick_bytes = uint64_t(info->max_block[0]) * info->max_block[1] *
                                 info->max_block[2] * (info->dtype == LV_DT_UINT16 ? 2u : 1u);
    lv_status st = launch_fbm_bricks(ctx, *info, *params, dperm.as<uint16_t>(),
                                     dids.as<uint64_t>(), n, static_cast<uint8_t*>(d_out),
                                     nullptr, brick_bytes, s);
    if (st != LV_OK)
        return st;
    /* the temporaries die at return */
    LV_CUDA(ctx, cudaStreamSynchronize(s));
    return LV_OK;
}

extern "C" lv_status lv_volume_create_fbm(lv_ctx* ctx, const lv_volume_info* info,
                                          const lv_fbm_params* params, uint32_t placement,
                                          uint32_t host_threads, lv_volume** out)
{
    if (!ctx || !info || !params || !out)
        return fail(ctx, LV_EINVAL, "null argument");
    if (info->dtype != LV_DT_UINT8 && info->dtype != LV_DT_UINT16)
        return fail(ctx, LV_EINVAL, "fBm volumes are uint8 or uint16");
    if (!valid_params(*params))
        return fail(ctx, LV_EINVAL, "fBm: 1..16 octaves, a positive frequency");
    if (placement == LV_FBM_HOST)
    {
        /* one brick per fetch thread (the generator is re-entrant) */
        FbmSource* src = new FbmSource{*info, *params, fbm_permutation(params->seed), 1u};
        lv_status st = lv_volume_create(ctx, info, fbm_source_get, src, out);
        if (st != LV_OK)
        {
            delete src;
            return st;
        }
        (*out)->user_free = fbm_source_free;
        st = lv_volume_set_fetch_threads(*out, std::min(host_threads, 64u));
        if (st != LV_OK)
        {
            lv_volume_destroy(*out);
            *out = nullptr;
        }
        return st;
    }
    if (placement != LV_FBM_DEVICE)
        return fail(ctx, LV_EINVAL, "unknown fBm placement");
    std::lock_guard<std::mutex> lock(ctx->mutex);
    LV_CUDA(ctx, cudaSetDevice(ctx->device));
    lv_volume* v = new lv_volume();
    v->ctx = ctx;
    v->info = *info;
    v->fbm = *params;
    v->kind = SRC_FBM_DEVICE;
    lv_status st = volume_init(ctx, v);
    if (st != LV_OK)
    {
        delete v;
        return st;
    }
    const std::vector<uint16_t> P = fbm_permutation(params->seed);
    if (v->d_perm.reserve(sizeof(uint16_t) * P.size()) != cudaSuccess ||
        cudaMemcpy(v->d_perm.ptr, P.data(), sizeof(uint16_t) * P.size(),
                   cudaMemcpyHostToDevice) != cudaSuccess)
    {
        delete v;
        return fail(ctx, LV_ENOMEM, "fBm permutation table");
    }
    *out = v;
    return LV_OK;
}
