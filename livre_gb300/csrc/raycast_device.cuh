/*
 * Device code of the ray cast shared by its translation units: view step
 * rule, voxel taps, interpolation, transfer function, ray set-up, brick
 * lookup and the march (raycast.cu describes the whole).
 */
#pragma once

#include "lv_runtime.h"

namespace lv
{
namespace
{
/* std::min / std::max semantics (first argument on ties), as the oracle. */
__device__ __forceinline__ float smin(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float smax(float a, float b) { return a < b ? b : a; }

/* nSamplesPerRay of a view from its finest rendered level (the rule of
 * step_body); every ray-cast CTA of lv_render evaluates it, the first one
 * also stores it for the frame statistics. */
__device__ __forceinline__ uint32_t view_samples(const RayView& V)
{
    uint32_t n = V.samples_fixed;
    if (n == 0)
    {
        const uint32_t ml = V.counters[FC_MAX_LEVEL];
        const uint32_t L = ml ? ml - 1u : 0u;
        const uint32_t shift = V.depth - L - 1u;
        if (V.step_policy == LV_STEP_HALF_VOXEL)
            n = (2u * V.max_voxel_dim) >> shift;
        else
            n = uint32_t(fmaxf(float(V.max_voxel_dim) / float(1u << shift), 512.0f));
        if (n == 0)
            n = 1;
    }
    return n;
}

__device__ __forceinline__ uint32_t frame_samples(const RayView& V)
{
    const uint32_t n = view_samples(V);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0)
        V.counters[FC_SAMPLES_PER_RAY] = n;
    return n;
}

/* Hardware base-2 exponential / logarithm (PTX ex2/lg2, approximate, FTZ). */
__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* One voxel as a float (the GL shader's conversion of an unsigned, signed or
 * float texel, fragRayCast.glsl:179-197; RayCastRenderer.cpp:236-277), read
 * only when `on` (else the value of zero bits). The load itself is
 * predicated (inline PTX), so a masked sample of the look-ahead march costs
 * no branch and touches no memory, and a sample's loads issue back to back:
 * with the voxel type a run-time switch, every tap was a branch and a load
 * waited for, and a 100^3 int16 thumbnail's ray cast took 404 us. */
template <int DT>
__device__ __forceinline__ float ldv_masked(const uint8_t* p, bool on)
{
#define LV_LD_MASKED(type)                                                                     \
    asm("{\n\t.reg .pred q;\n\t.reg .u64 g;\n\tcvta.to.global.u64 g, %1;\n\t"                   \
        "setp.ne.b32 q, %2, 0;\n\t@q ld.global.nc." type " %0, [g];\n\t}"                      \
        : "+r"(v)                                                                              \
        : "l"(p), "r"(uint32_t(on)))
    uint32_t v = 0;
    switch (DT)
    {
    case LV_DT_UINT8: LV_LD_MASKED("u8"); return float(v);
    case LV_DT_UINT16: LV_LD_MASKED("u16"); return float(v);
    case LV_DT_INT8: LV_LD_MASKED("s8"); return float(int32_t(v));
    case LV_DT_INT16: LV_LD_MASKED("s16"); return float(int32_t(v));
    case LV_DT_UINT32: LV_LD_MASKED("u32"); return __uint2float_rn(v);
    case LV_DT_INT32: LV_LD_MASKED("u32"); return __int2float_rn(int32_t(v));
    default: LV_LD_MASKED("u32"); return __uint_as_float(v);
    }
#undef LV_LD_MASKED
}

/* Bytes of one voxel. */
__host__ __device__ constexpr int voxel_bytes(int dt)
{
    return dt == LV_DT_UINT8 || dt == LV_DT_INT8     ? 1
           : dt == LV_DT_UINT16 || dt == LV_DT_INT16 ? 2
                                                     : 4;
}

/* The two voxel quads of a trilinear sample in a uint8 quad-layout brick
 * (quad_layout: voxels (x, y), (x + 1, y), (x, y + 1), (x + 1, y + 1) in
 * bytes 0 to 3), slices z and z + 1 at byte offsets 0 and dz from p, read
 * only when `on` under one predicate; when !on the registers hold whatever
 * they held (any byte converts to a finite float, and the sample is
 * masked). */
__device__ __forceinline__ void ld_quads2(const uint8_t* p, uint32_t dz, bool on,
                                          uint32_t (&q)[2])
{
    asm("{\n\t.reg .pred q;\n\t.reg .u64 g, h;\n\tcvta.to.global.u64 g, %2;\n\t"
        "cvt.u64.u32 h, %4;\n\tadd.u64 h, g, h;\n\t"
        "setp.ne.b32 q, %3, 0;\n\t"
        "@q ld.global.nc.u32 %0, [g];\n\t"
        "@q ld.global.nc.u32 %1, [h];\n\t}"
        : "=r"(q[0]), "=r"(q[1])
        : "l"(p), "r"(uint32_t(on)), "r"(dz));
}

/* The same with the slice pitch DZ an immediate offset (fixed-pitch
 * kernels). */
template <int DZ>
__device__ __forceinline__ void ld_quads2(const uint8_t* p, bool on, uint32_t (&q)[2])
{
    asm("{\n\t.reg .pred q;\n\t.reg .u64 g;\n\tcvta.to.global.u64 g, %2;\n\t"
        "setp.ne.b32 q, %3, 0;\n\t"
        "@q ld.global.nc.u32 %0, [g];\n\t"
        "@q ld.global.nc.u32 %1, [g+%4];\n\t}"
        : "=r"(q[0]), "=r"(q[1])
        : "l"(p), "r"(uint32_t(on)), "n"(DZ));
}

/* The voxels a sample reads and its interpolation weights; loaded one
 * sample ahead of the compositing (march) so that the loads of the next
 * sample are in flight while the current one is composited. The trilinear
 * taps of the fixed-pitch voxel-quad kernels (raw_taps) stay as the two
 * loaded quad words until the sample is composited: two registers per tap
 * set instead of eight. */
template <int FILTER>
struct Taps
{
    static constexpr int N = FILTER == LV_FILTER_TRILINEAR ? 8 : 1;
    float c[N];
    uint32_t q[2]; /* raw_taps: the quads of slices z and z + 1 */
    float fx, fy, fz;
};

template <int DT, int FILTER, int EDGE>
__host__ __device__ constexpr bool raw_taps()
{
    return DT == LV_DT_UINT8 && FILTER == LV_FILTER_TRILINEAR &&
           quad_layout(DT, EDGE > 1 ? EDGE : 0);
}

/* The view constants the per-sample steps read (the transfer function and
 * its coordinate map, the early-termination opacity, the last trilinear
 * base voxel). A kernel that renders one view passes its RayView parameter
 * itself (constant-bank operands); the persistent batch kernel, whose view
 * changes from tile to tile, passes this register copy instead of reading
 * its shared-memory view on every sample. */
struct HotView
{
    const float4* tf;
    float tf_mul, tf_add, tf_last, early;
    uint32_t max_base;
};

__device__ __forceinline__ HotView hot_view(const RayView& V)
{
    HotView h;
    h.tf = V.tf;
    h.tf_mul = V.tf_mul;
    h.tf_add = V.tf_add;
    h.tf_last = V.tf_last;
    h.early = V.early;
    h.max_base = V.max_base;
    return h;
}

/* Voxels around slot coordinate s (nearest: s = local position; trilinear:
 * s = local position - 0.5, texel centres on integers). EDGE = 1 clamps every
 * tap to the brick (GL_CLAMP_TO_EDGE, needed without overlap); EDGE = 0 uses
 * one base address and offsets to the other taps, valid when every overlap
 * >= 1; EDGE = n > 1 is EDGE = 0 for bricks of n x n voxels in x and y (the
 * row and slice pitches become immediate offsets of one pointer). */
template <int DT, int FILTER, int EDGE, class HV>
__device__ __forceinline__ void load_taps(const RayView& V, const HV& H, const uint8_t* brick,
                                          const float s[3], Taps<FILTER>& T, bool on)
{
    /* the voxels are read only when `on` (the sample has data) */
    auto ld = [&](const uint8_t* q) { return ldv_masked<DT>(q, on); };
    constexpr int NX = EDGE > 1 ? EDGE : 0;
    /* voxel quads (quad_layout): known from the pitch for fixed-pitch
     * kernels, else the view's flag */
    const bool quads = DT == LV_DT_UINT8 && (NX ? quad_layout(DT, NX) : V.quads != 0);
    /* bytes per stored voxel element */
    const int bpv = quads ? 4 : voxel_bytes(DT);
    const int n0 = NX ? NX : int(V.N[0]), n1 = NX ? NX : int(V.N[1]), n2 = int(V.N[2]);
    if (FILTER == LV_FILTER_NEAREST)
    {
        const int x = min(max(int(floorf(s[0])), 0), n0 - 1);
        const int y = min(max(int(floorf(s[1])), 0), n1 - 1);
        const int z = min(max(int(floorf(s[2])), 0), n2 - 1);
        T.c[0] = ld(brick + ((z * n1 + y) * n0 + x) * bpv);
        return;
    }
    /* floor by adding 2^23 rounding down (exact for |s| < 2^22), no
     * conversion instruction; x and y as one packed pair */
    const float2 kM = make_float2(8388608.0f, 8388608.0f);
    const float2 sxy = make_float2(s[0], s[1]);
    const float2 fxy0 = __fadd2_rn(__fadd2_rd(sxy, kM), make_float2(-8388608.0f, -8388608.0f));
    const float fx0 = fxy0.x, fy0 = fxy0.y;
    const float fz0 = __fadd_rd(s[2], 8388608.0f) - 8388608.0f;
    const float2 fxy = __ffma2_rn(fxy0, make_float2(-1.0f, -1.0f), sxy); /* s - floor(s) */
    T.fx = fxy.x;
    T.fy = fxy.y;
    T.fz = s[2] - fz0;
    const int ix = int(fx0), iy = int(fy0), iz = int(fz0);
    if (EDGE == 1)
    {
        const int x0 = min(max(ix, 0), n0 - 1), x1 = min(max(ix + 1, 0), n0 - 1);
        const int y0 = min(max(iy, 0), n1 - 1), y1 = min(max(iy + 1, 0), n1 - 1);
        const int z0 = min(max(iz, 0), n2 - 1), z1 = min(max(iz + 1, 0), n2 - 1);
        const int r00 = (z0 * n1 + y0) * n0, r01 = (z0 * n1 + y1) * n0;
        const int r10 = (z1 * n1 + y0) * n0, r11 = (z1 * n1 + y1) * n0;
        T.c[0] = ld(brick + (r00 + x0) * bpv);
        T.c[1] = ld(brick + (r00 + x1) * bpv);
        T.c[2] = ld(brick + (r01 + x0) * bpv);
        T.c[3] = ld(brick + (r01 + x1) * bpv);
        T.c[4] = ld(brick + (r10 + x0) * bpv);
        T.c[5] = ld(brick + (r10 + x1) * bpv);
        T.c[6] = ld(brick + (r11 + x0) * bpv);
        T.c[7] = ld(brick + (r11 + x1) * bpv);
    }
    else
    {
        /* every overlap >= 1: for a sample in cell c the slot coordinate is in
         * [O - 1/2, O + B - 1/2], so the base voxel is in [0, N - 2] on each
         * axis and all eight taps are in the slot. One unsigned clamp of the
         * linear base keeps any tap inside the slot whatever the inputs. */
        const uint32_t base =
            min(__float2uint_rz(fmaf(fmaf(fz0, float(n1), fy0), float(n0), fx0)), H.max_base);
        const int dy = n0 * bpv, dz = n0 * n1 * bpv;
        const uint8_t* p00 = brick + base * bpv;
        const uint8_t* p01 = p00 + dy;
        const uint8_t* p10 = p00 + dz;
        const uint8_t* p11 = p10 + dy;
        if (raw_taps<DT, FILTER, EDGE>())
        {
            /* the quads of slices z and z + 1, kept raw until the sample is
             * composited. The address is formed as a 64-bit product: the same
             * address as p00's 32-bit one compiled to a schedule that ray
             * casts the 2048^3 / 1080p orbit 11 % slower (0.259 against
             * 0.232 ms). */
            ld_quads2<4 * NX * NX>(brick + uint64_t(base) * 4u, on, T.q);
            return;
        }
        if (DT == LV_DT_UINT8 && quads)
        {
            /* the quad layout in a generic-pitch kernel: two quad loads,
             * converted here */
            uint32_t q[2];
            ld_quads2(p00, uint32_t(dz), on, q);
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                T.c[k] = float((q[0] >> (8 * k)) & 0xFFu);
                T.c[4 + k] = float((q[1] >> (8 * k)) & 0xFFu);
            }
            return;
        }
        T.c[0] = ld(p00);
        T.c[1] = ld(p00 + bpv);
        T.c[2] = ld(p01);
        T.c[3] = ld(p01 + bpv);
        T.c[4] = ld(p10);
        T.c[5] = ld(p10 + bpv);
        T.c[6] = ld(p11);
        T.c[7] = ld(p11 + bpv);
    }
}

/* Trilinear weights applied x, then y, then z (the oracle's order):
 *   a0 = lerp(c0, c1, fx)  a1 = lerp(c2, c3, fx)  a2 = lerp(c4, c5, fx)
 *   a3 = lerp(c6, c7, fx)  b0 = lerp(a0, a1, fy)  b1 = lerp(a2, a3, fy)
 *   v  = lerp(b0, b1, fz), lerp(a, b, f) = fma(b - a, f, a).
 * Independent lerps run as pairs in packed FP32 instructions (FFMA2: one
 * issue for two IEEE fused multiply-adds, each rounded as the scalar one;
 * b - a as fma(a, -1, b) is the same single rounding), paired so that every
 * result lands in the register pair the next stage reads: (a0, a2) and
 * (a1, a3), then (b0, b1). */
template <int FILTER, bool RAW>
__device__ __forceinline__ float interp(const Taps<FILTER>& T)
{
    if (FILTER == LV_FILTER_NEAREST)
        return T.c[0];
    const float2 m1 = make_float2(-1.0f, -1.0f);
    const float2 fx = make_float2(T.fx, T.fx);
    float2 a02, a13;
    if (RAW)
    {
        /* a voxel byte b placed by a byte permute into the mantissa of 2^23
         * is the float 2^23 + b (exact, no conversion instruction): the
         * difference of two such floats is hi - lo exactly, and subtracting
         * 2^23 gives lo exactly, so every lerp sees the values above */
        auto bt = [](uint32_t q, uint32_t k) {
            return __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7440u + k));
        };
        const float2 mM = make_float2(-8388608.0f, -8388608.0f);
        /* quad bytes 0..3: c0..c3 of slice z (T.q[0]), c4..c7 of z + 1 */
        const float2 lo0 = make_float2(bt(T.q[0], 0), bt(T.q[1], 0));
        const float2 hi0 = make_float2(bt(T.q[0], 1), bt(T.q[1], 1));
        const float2 lo1 = make_float2(bt(T.q[0], 2), bt(T.q[1], 2));
        const float2 hi1 = make_float2(bt(T.q[0], 3), bt(T.q[1], 3));
        a02 = __ffma2_rn(__ffma2_rn(lo0, m1, hi0), fx, __fadd2_rn(lo0, mM));
        a13 = __ffma2_rn(__ffma2_rn(lo1, m1, hi1), fx, __fadd2_rn(lo1, mM));
    }
    else
    {
        const float2 lo0 = make_float2(T.c[0], T.c[4]), hi0 = make_float2(T.c[1], T.c[5]);
        const float2 lo1 = make_float2(T.c[2], T.c[6]), hi1 = make_float2(T.c[3], T.c[7]);
        a02 = __ffma2_rn(__ffma2_rn(lo0, m1, hi0), fx, lo0);
        a13 = __ffma2_rn(__ffma2_rn(lo1, m1, hi1), fx, lo1);
    }
    const float2 b01 = __ffma2_rn(__ffma2_rn(a02, m1, a13), make_float2(T.fy, T.fy), a02);
    return fmaf(b01.y - b01.x, T.fz, b01.x);
}

/* Linear, clamp-to-edge lookup of the transfer function at voxel value v
 * (texel coordinate v * tf_mul + tf_add = density * tfn - 1/2), stored as
 * interleaved (value_i, value_{i+1} - value_i) pairs (last difference 0).
 * Clamping the coordinate to [0, tfn - 1] before splitting it gives the
 * same texel pair and weight as clamping the texel index after. */
template <int TFS, class HV>
__device__ __forceinline__ float4 tf_lookup(const HV& H, float v)
{
    const float s = fminf(fmaxf(fmaf(v, H.tf_mul, H.tf_add), 0.0f), H.tf_last);
    /* floor(s) (s in [0, tf_last]) by adding 2^23 rounding down: its bits
     * carry the integer, no conversion instruction */
    const float y = __fadd_rd(s, 8388608.0f);
    const int i0 = int(__float_as_uint(y) - 0x4B000000u);
    const float f = s - (y - 8388608.0f);
    /* TFS: the table is in shared memory (generic loads); else read-only
     * global memory, the texel pair's 32 bytes (value, difference) in one
     * 256-bit load: the table is a device allocation, so every pair is
     * 32-byte aligned */
    const float4* e = H.tf + 2 * i0;
    float4 a, b;
    if (TFS)
    {
        a = e[0];
        b = e[1];
    }
    else
        asm("{\n\t.reg .u64 g;\n\tcvta.to.global.u64 g, %8;\n\t"
            "ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [g];\n\t}"
            : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z),
              "=f"(b.w)
            : "l"(e));
    /* value + difference * f per channel, two channels per FFMA2 */
    const float2 f2 = make_float2(f, f);
    const float2 rg = __ffma2_rn(make_float2(b.x, b.y), f2, make_float2(a.x, a.y));
    const float2 ba = __ffma2_rn(make_float2(b.z, b.w), f2, make_float2(a.z, a.w));
    return make_float4(rg.x, rg.y, ba.x, ba.y);
}

__device__ __forceinline__ float Md(const float* m, int r, int c)
{
    return m[c * 4 + r];
}

struct RayGeom
{
    float dir[3];
    float tg, tlo, thi;
    bool hit;
};

/* Pixel (px, py) of the rendered rect as an index into the frame. */
__device__ __forceinline__ uint64_t frame_index(const RayView& V, uint32_t px, uint32_t py)
{
    return uint64_t(py + V.y0) * V.FW + (px + V.x0);
}

/* Ray through the centre of pixel (px, py) of the rendered rect (frame pixel
 * (x0 + px, y0 + py)); FP32 IEEE ops in fixed order. A pixel outside the
 * view's conservative screen rectangle of the volume's box (V.cull) misses
 * the box: it returns no hit without the set-up arithmetic, as the full
 * computation would (about 85 % of a 1080p orbit frame's pixels). */
__device__ __forceinline__ RayGeom ray_setup(const RayView& V, uint32_t px,
                                             uint32_t py)
{
    RayGeom g;
    const uint32_t fx = px + V.x0, fy = py + V.y0;
    if (fx < V.cull[0] || fx >= V.cull[2] || fy < V.cull[1] || fy >= V.cull[3])
    {
        g.dir[0] = g.dir[1] = g.dir[2] = 0.0f;
        g.tg = g.tlo = g.thi = 0.0f;
        g.hit = false;
        return g;
    }
    const float nx =
        __fsub_rn(__fdiv_rn(__fmul_rn(__fadd_rn(__uint2float_rn(px + V.x0), 0.5f), 2.0f),
                            __uint2float_rn(V.FW)),
                  1.0f);
    const float ny =
        __fsub_rn(__fdiv_rn(__fmul_rn(__fadd_rn(__uint2float_rn(py + V.y0), 0.5f), 2.0f),
                            __uint2float_rn(V.FH)),
                  1.0f);
    float e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        e[i] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(Md(V.inv_p, i, 0), nx),
                                             __fmul_rn(Md(V.inv_p, i, 1), ny)),
                                   __fmul_rn(Md(V.inv_p, i, 2), -1.0f)),
                         __fmul_rn(Md(V.inv_p, i, 3), 1.0f));
    const float ep[3] = {__fdiv_rn(e[0], e[3]), __fdiv_rn(e[1], e[3]),
                         __fdiv_rn(e[2], e[3])};
    float d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const float pw =
            __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(Md(V.inv_mv, i, 0), ep[0]),
                                          __fmul_rn(Md(V.inv_mv, i, 1), ep[1])),
                                __fmul_rn(Md(V.inv_mv, i, 2), ep[2])),
                      Md(V.inv_mv, i, 3));
        d[i] = __fsub_rn(pw, V.eye[i]);
    }
    const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]),
                                                     __fmul_rn(d[1], d[1])),
                                           __fmul_rn(d[2], d[2])));
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g.dir[i] = __fdiv_rn(d[i], len);
    const float lenE = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(ep[0], ep[0]),
                                                      __fmul_rn(ep[1], ep[1])),
                                            __fmul_rn(ep[2], ep[2])));
    const float nz = __fdiv_rn(ep[2], lenE);
    const float tnp = __fdiv_rn(-V.nearp, nz);
    float tmin[3], tmax[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const float di = g.dir[i] == 0.0f ? 1e-10f : g.dir[i];
        const float inv = __fdiv_rn(1.0f, di);
        const float tb = __fmul_rn(inv, __fsub_rn(V.gmin[i], V.eye[i]));
        const float tt = __fmul_rn(inv, __fsub_rn(V.gmax[i], V.eye[i]));
        tmin[i] = smin(tt, tb);
        tmax[i] = smax(tt, tb);
    }
    const float t0 = smax(smax(tmin[0], tmin[1]), smax(tmin[0], tmin[2]));
    const float t1 = smin(smin(tmax[0], tmax[1]), smin(tmax[0], tmax[2]));
    g.hit = t0 <= t1;
    g.tg = t0;
    float tlo = smax(t0, tnp);
    float thi = t1;
    for (uint32_t c = 0; c < V.n_clip; ++c)
    {
        const float* cp = V.clip[c];
        float rn = __fadd_rn(__fadd_rn(__fmul_rn(g.dir[0], cp[0]), __fmul_rn(g.dir[1], cp[1])),
                             __fmul_rn(g.dir[2], cp[2]));
        if (rn == 0.0f)
            rn = 1e-10f;
        const float ne = __fadd_rn(__fadd_rn(__fmul_rn(cp[0], V.eye[0]), __fmul_rn(cp[1], V.eye[1])),
                                   __fmul_rn(cp[2], V.eye[2]));
        const float t = __fdiv_rn(-__fadd_rn(ne, cp[3]), rn);
        if (rn > 0.0f)
            tlo = smax(tlo, t);
        else
            thi = smin(thi, t);
    }
    g.tlo = tlo;
    g.thi = thi;
    return g;
}

/* State of one ray between two samples, so that a lane can take a number of
 * samples, stop, and go on later (the refill kernels below). */
struct RayState
{
    float dir[3];
    float tg, thi;
    float kf;            /* index of the next sample (exact in FP32 below 2^24) */
    float kf_safe;       /* samples up to this index stay in the current brick */
    uint32_t err;        /* FC_ERROR value to report when the ray ends (0: none) */
    float4 dst;
    uint32_t entry;      /* leaf entry of the current brick (or empty cell) */
    const uint8_t* brick;
    /* slot coordinate of a sample of the brick: sc = fma(t, sa, sb), the
     * composition of the position, cell and slot maps (a few ulp from the
     * oracle's three-FMA chain; which brick a sample reads is exact) */
    float sa[3], sb[3];
};

/* First sample on the global grid at or after tlo; false: no sample. */
__device__ __forceinline__ bool ray_begin(const RayGeom& g, float step, RayState& r)
{
    r.dst = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!g.hit || !(g.tlo <= g.thi))
        return false;
    int k = 0;
    if (g.tlo > g.tg)
        k = int(ceilf(__fdiv_rn(__fsub_rn(g.tlo, g.tg), step)));
    r.kf = __int2float_rn(k);
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        r.dir[a] = g.dir[a];
        r.sa[a] = 0.f;
        r.sb[a] = 0.f;
    }
    r.tg = g.tg;
    r.thi = g.thi;
    r.kf_safe = -1.0f;
    r.err = 0u;
    r.entry = kLeafEmpty;
    r.brick = nullptr;
    return true;
}

/* Sample position in leaf-cell units at ray parameter t: single-rounding
 * FMAs in a fixed order (the CPU oracle evaluates the same fmaf chain). */
__device__ __forceinline__ void sample_cell_coord(const RayView& V, const RayState& r, float t,
                                                  float f[3])
{
#pragma unroll
    for (int a = 0; a < 3; ++a)
        f[a] = fmaf(fmaf(r.dir[a], t, V.eye[a]), V.gscale[a], V.goff[a]);
}

/* Leaf cell of a sample at cell coordinate f on one axis (dims or more:
 * outside the octree). The sample's parameter is in [tnearGlobal,
 * tfarGlobal), so it lies in the volume's box: a cell index rounded one past
 * the box's face (a sample on the entry or exit face, which the reference
 * shader takes at tnear = tnearGlobal, fragRayCast.glsl:142-147) is the face
 * cell. The low face is the box's on every axis (f = 0); the high face only
 * on axes with the most cells (cell_hi): shorter axes end inside the box, as
 * the node boxes of LODNode.cpp:30-64 (cell side worldSize / maxBricks) do.
 * The floor of the clamped coordinate (below 2^22) comes from the low bits of
 * its sum with 2^23 rounded down. */
__device__ __forceinline__ uint32_t face_cell(float f, float cell_hi)
{
    return __float_as_uint(__fadd_rd(fminf(fmaxf(f, 0.0f), cell_hi), 8388608.0f)) - 0x4B000000u;
}

/* The slow path of a sample (index r.kf, position f) that leaves the range
 * known to lie in the current brick: finds its leaf cell (face_cell), the
 * brick there, and how far the ray stays in that brick. False: the sample
 * is outside the octree.
 *
 * The cell of a sample is monotone in its index along each axis (t, the
 * position and f are monotone single-rounding functions of it, and floor is
 * monotone), so if the sample at index k lies in the brick's cube of leaf
 * cells, so does every sample between this one and k. k is the estimated
 * last sample before the exit (or the one before it), checked with the
 * exact per-sample position against the cube's bounds; samples up to
 * r.kf_safe then skip the lookup and take the same brick the per-sample
 * lookup would.
 *
 * The lanes of a warp cross a brick's face in different iterations, so the
 * lookup runs several times per face and warp and its instructions count: it
 * is written without conversions (integers pass through the mantissa of
 * 2^23), with one reciprocal per axis and on constants of the view: a 256^3
 * volume in 32^3 bricks at 512 x 512 ray casts in 175 us (196 with
 * conversions and two divisions per axis), 64^3 bricks with one voxel per
 * pixel at 1280 x 720 in 627 us (704). */
template <int FILTER>
__device__ __forceinline__ bool locate(const RayView& V, RayState& r, float step, const float f[3])
{
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        c[a] = face_cell(f[a], V.cell_hi[a]);
    r.kf_safe = r.kf; /* this sample only, unless shown otherwise below */
    if (!(c[0] < V.dims[0] && c[1] < V.dims[1] && c[2] < V.dims[2]))
        return false;
    uint32_t entry = __ldg(V.leaf + (c[2] * V.dims[1] + c[1]) * V.dims[0] + c[0]);
    if (entry != kLeafEmpty && ((entry & kLeafSlotMask) + V.brick_units > V.pool_units ||
                                (entry >> kLeafSlotBits) > V.Lf))
    {
        /* entry outside the pool: reported when the ray ends, so that the
         * sample loop stores nothing to memory */
        r.err = 3u;
        entry = kLeafEmpty;
    }
    r.entry = entry;
    /* an empty cell spans one leaf cell; a brick at level L spans 2^(Lf-L) */
    const uint32_t sh = entry == kLeafEmpty ? 0u : V.Lf - (entry >> kLeafSlotBits);
    const float side = __uint_as_float((127u + sh) << 23);     /* 2^sh */
    const float inv_side = __uint_as_float((127u - sh) << 23); /* 2^-sh */
    if (entry != kLeafEmpty)
        r.brick = V.pool + uint64_t(entry & kLeafSlotMask) * kSlotUnit;
    float lo[3], hi[3], tx = 3.0e38f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        /* the cube's first cell, exact in FP32 */
        const float first =
            __uint_as_float(((c[a] >> sh) << sh) + 0x4B000000u) - 8388608.0f;
        const float fd = r.dir[a] * V.gscale[a];
        if (entry != kLeafEmpty)
        {
            /* slot coordinate = f * vs + off (vs, off exact); composed with
             * f = (eye + dir * t) * gscale + goff into one map of t */
            const float vs = V.Bf[a] * inv_side;
            r.sa[a] = fd * vs;
            r.sb[a] = fmaf(V.f0[a], vs, fmaf(-first, vs, V.Oh[a]));
        }
        /* the positions face_cell puts in the cube */
        lo[a] = first == 0.0f ? -INFINITY : first;
        hi[a] = first + side >= float(V.dims[a]) ? V.cube_end[a] : first + side;
        /* estimated parameter where the ray leaves it on this axis */
        const float te = __fdividef((fd > 0.0f ? hi[a] : lo[a]) - V.f0[a], fd);
        tx = fd != 0.0f ? fminf(tx, te) : tx;
    }
    float ke = fminf(floorf(__fdividef(tx - r.tg, step)), 16777215.0f);
#pragma unroll 1
    for (int attempt = 0; attempt < 2 && ke > r.kf; ++attempt, ke -= 1.0f)
    {
        float g[3];
        sample_cell_coord(V, r, fmaf(ke, step, r.tg), g);
        if (g[0] >= lo[0] && g[0] < hi[0] && g[1] >= lo[1] && g[1] < hi[1] && g[2] >= lo[2] &&
            g[2] < hi[2])
        {
            r.kf_safe = ke;
            break;
        }
    }
    return true;
}

/* Takes the ray's sample r.kf and advances it by STRIDE samples, with one divergent
 * region, the brick lookup where the ray leaves its safe range; false once
 * the ray has left its segment. The sample's voxels are read into T only
 * when it has data (`valid`: inside the segment and in a rendered brick, not
 * outside the octree or in a cell no brick covers), by predicated loads, so
 * a sample without data costs no branch. */
template <int DT, int FILTER, int EDGE, int STRIDE = 1, class HV>
__device__ __forceinline__ bool fetch_sample(const RayView& V, const HV& H, RayState& r, float step,
                                         Taps<FILTER>& T, bool& valid)
{
    const float t = fmaf(r.kf, step, r.tg);
    const bool live = t < r.thi;
    if (live && !(r.kf <= r.kf_safe))
    {
        float f[3];
        sample_cell_coord(V, r, t, f);
        if (!locate<FILTER>(V, r, step, f))
            r.entry = kLeafEmpty; /* outside the octree: this sample has no data */
    }
    r.kf += float(STRIDE);
    valid = live && r.entry != kLeafEmpty;
    float sc[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        sc[a] = fmaf(t, r.sa[a], r.sb[a]);
    load_taps<DT, FILTER, EDGE>(V, H, r.brick, sc, T, valid);
    return live;
}

/* Transfer function, opacity correction and front-to-back blending of one
 * sample (fragRayCast.glsl:103-111); false once the early-termination
 * opacity is reached. A sample without data (!valid) is blended with opacity
 * 0 (the colour and opacity stay bit for bit as they were) and not counted,
 * so the march needs no branch around it. */
template <int FILTER, int TFS, bool RAW, class HV>
__device__ __forceinline__ bool composite_sample(const HV& H, RayState& r, float ac,
                                                 const Taps<FILTER>& T, bool valid,
                                                 uint32_t& nsamp)
{
    const float4 src = tf_lookup<TFS>(H, interp<FILTER, RAW>(T));
    const float am = fminf(src.w, 1.0f - 1.0f / 256.0f);
    const float alpha = valid ? 1.0f - ex2_approx(ac * lg2_approx(1.0f - am)) : 0.0f;
    const float w = alpha * (1.0f - r.dst.w);
    r.dst.x = fmaf(src.x, w, r.dst.x);
    r.dst.y = fmaf(src.y, w, r.dst.y);
    r.dst.z = fmaf(src.z, w, r.dst.z);
    r.dst.w = fmaf(alpha, 1.0f - r.dst.w, r.dst.w);
    nsamp += valid ? 1u : 0u;
    return !(r.dst.w > H.early);
}

/* One sample of the ray, fetched and composited with one tap set: false
 * once the ray has ended or reached the early-termination opacity. */
template <int DT, int FILTER, int TFS, int EDGE, class HV>
__device__ __forceinline__ bool ray_step(const RayView& V, const HV& H, RayState& r, float step,
                                         float ac, uint32_t& nsamp)
{
    Taps<FILTER> T;
    bool valid;
    const bool live = fetch_sample<DT, FILTER, EDGE>(V, H, r, step, T, valid);
    const bool cont =
        composite_sample<FILTER, TFS, raw_taps<DT, FILTER, EDGE>()>(H, r, ac, T, valid, nsamp);
    return live && cont;
}

/* A ray has ended: report an index check it failed. */
__device__ __forceinline__ void flush_error(const RayView& V, const RayState& r)
{
    if (r.err)
        atomicExch(&V.counters[FC_ERROR], r.err);
}

/* Colour a ray starts from: the frame so far in a later pass of a
 * multi-pass frame (RenderPipeline.cpp:92-158 composites every pass into
 * the same render texture), else transparent black. */
__device__ __forceinline__ float4 initial_dst(const RayView& V, uint32_t px, uint32_t py)
{
    return V.accumulate ? V.out[frame_index(V, px, py)] : make_float4(0.f, 0.f, 0.f, 0.f);
}

/* The whole ray. LOOKAHEAD = 1 loads the voxels of sample k + 1 before
 * sample k is composited, so the two latency chains overlap (a lone long
 * ray runs faster; more registers per thread). Samples, values and the
 * compositing order are those of ray_step either way; after an early
 * termination the loads of one extra sample are dropped. */
template <int DT, int FILTER, int TFS, int EDGE, int LOOKAHEAD, class HV>
__device__ float4 march(const RayView& V, const HV& H, const RayGeom& g, float step,
                        float ac, uint32_t& nsamp,
                        float4 init = make_float4(0.f, 0.f, 0.f, 0.f))
{
    RayState r;
    if (!ray_begin(g, step, r) || init.w > H.early)
        return init;
    r.dst = init;
    if (!LOOKAHEAD)
    {
        while (ray_step<DT, FILTER, TFS, EDGE>(V, H, r, step, ac, nsamp))
        {
        }
        flush_error(V, r);
        return r.dst;
    }
    /* two tap sets in turn (no copy of the taps between samples): fetch the
     * next sample into one while the other is composited. A sample without
     * data is fetched and composited masked, so each sample has one
     * divergent region (a brick lookup) and one loop exit. */
    constexpr bool RAW = raw_taps<DT, FILTER, EDGE>();
    Taps<FILTER> T0, T1;
    bool v0, v1;
    bool live0 = fetch_sample<DT, FILTER, EDGE>(V, H, r, step, T0, v0);
    while (live0)
    {
        const bool live1 = fetch_sample<DT, FILTER, EDGE>(V, H, r, step, T1, v1);
        if (!(composite_sample<FILTER, TFS, RAW>(H, r, ac, T0, v0, nsamp) && live1))
            break;
        live0 = fetch_sample<DT, FILTER, EDGE>(V, H, r, step, T0, v0);
        if (!composite_sample<FILTER, TFS, RAW>(H, r, ac, T1, v1, nsamp))
            break;
    }
    flush_error(V, r);
    return r.dst;
}

/* The ray cast of a view whose frame will be rendered again
 * (RayView::skip_if_missing): every block of the launch returns at once. */
__device__ __forceinline__ bool skip_frame(const RayView& V)
{
    return V.skip_if_missing &&
           *static_cast<const volatile uint32_t*>(V.counters + FC_MISSING) != 0u;
}

/* One CTA per tile: block i renders tile order[i] (or tile i). */
template <int DT, int FILTER, int EDGE, int LA>
__device__ __forceinline__ void cast_tile(const RayView& V, uint32_t tile_w, uint32_t tile_h,
                                          const uint32_t* __restrict__ order)
{
    if (skip_frame(V))
        return;
    const uint32_t n = frame_samples(V);
    const float step = __fdiv_rn(1.0f, __uint2float_rn(n));
    const float ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    const uint32_t tiles_x = (V.W + tile_w - 1) / tile_w;
    const uint32_t tile = order ? order[blockIdx.x] : blockIdx.x;
    const uint32_t px = (tile % tiles_x) * tile_w + threadIdx.x % tile_w;
    const uint32_t py = (tile / tiles_x) * tile_h + threadIdx.x / tile_w;
    uint32_t nsamp = 0;
    if (px < V.W && py < V.H)
    {
        const RayGeom g = ray_setup(V, px, py);
        V.out[frame_index(V, px, py)] =
            march<DT, FILTER, 0, EDGE, LA>(V, V, g, step, ac, nsamp, initial_dst(V, px, py));
    }
    unsigned long long sum = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31u) == 0 && sum)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), sum);
}

template <int DT, int FILTER, int EDGE, int LA>
__global__ void __launch_bounds__(256)
    raycast_tiles_kernel(const __grid_constant__ RayView V, uint32_t tile_w, uint32_t tile_h,
                         const uint32_t* __restrict__ order)
{
    cast_tile<DT, FILTER, EDGE, LA>(V, tile_w, tile_h, order);
}

/* The same compiled for two resident blocks of 256 threads: 74 registers
 * instead of 64 (uint16, trilinear, look-ahead), so 12 blocks of 64 threads
 * share an SM's L1 instead of 16 (roomy_l1 chooses). */
template <int DT, int FILTER, int EDGE, int LA>
__global__ void __launch_bounds__(256, 2)
    raycast_tiles_roomy_kernel(const __grid_constant__ RayView V, uint32_t tile_w,
                               uint32_t tile_h, const uint32_t* __restrict__ order)
{
    cast_tile<DT, FILTER, EDGE, LA>(V, tile_w, tile_h, order);
}

/* ---------------------------------------------------------- split rays
 * S lanes of a warp share a ray: lane j takes its samples j, j + S, j + 2S,
 * ... In each iteration they fetch, interpolate and classify S consecutive
 * samples side by side and exchange the colours and opacities through shared
 * memory; lane j then blends channel j % 4 of all S, in sample order. So the
 * samples, their values, the blending order and the roundings are march()'s
 * (image and sample count bit for bit), while a ray's chain of dependent
 * loads is S times shorter, a frame has S times more warps, and the lanes of
 * a warp read S consecutive positions of 32 / S rays instead of one position
 * of 32 rays, which touches fewer cache lines where a pixel spans a voxel or
 * more (uint8 quads, one voxel per pixel, S = 4: 3.4 L1 wavefronts per load
 * request against 6.6).
 *
 * The price is the exchange and S blends instead of one, about 60
 * instructions on 85 with S = 4, so a frame of many rays whose issue slots
 * are busy is faster with one lane per ray: split_lanes (raycast.cu) chooses. */
template <int S>
struct RayGroup
{
    /* a ray's row of the exchange buffer: 4 planes (red, green, blue,
     * opacity) of S values, padded so that a warp's plane write (32 / S rows)
     * hits 32 banks */
    static constexpr int kRow = S == 4 ? 20 : 4 * S + 8;
    float c; /* this lane's channel, blended so far (lanes 3 mod 4: blue again) */
    float a; /* the opacity, in every lane */

    __device__ __forceinline__ static uint32_t plane(uint32_t j) { return min(j & 3u, 2u) * S; }

    __device__ __forceinline__ void blend(float v, float alpha)
    {
        /* composite_sample's blend */
        const float w = alpha * (1.0f - a);
        c = fmaf(v, w, c);
        a = fmaf(alpha, 1.0f - a, a);
    }

    /* blends a row; true, with the group as before, when the opacity passed
     * `early` on the way */
    __device__ __forceinline__ bool blend_row(const float* row, uint32_t j, float early)
    {
        const RayGroup was = *this;
        bool stop = false;
#pragma unroll
        for (int q = 0; q < S; q += 4)
        {
            const float4 alpha = *reinterpret_cast<const float4*>(row + 3 * S + q);
            const float4 v = *reinterpret_cast<const float4*>(row + plane(j) + q);
            blend(v.x, alpha.x);
            stop = stop || a > early;
            blend(v.y, alpha.y);
            stop = stop || a > early;
            blend(v.z, alpha.z);
            stop = stop || a > early;
            blend(v.w, alpha.w);
            stop = stop || a > early;
        }
        if (stop)
            *this = was;
        return stop;
    }

    /* blends a row up to and with the sample that passes `early` and returns
     * that sample's place (the last place if none does) */
    __device__ __forceinline__ uint32_t blend_to_stop(const float* row, uint32_t j, float early)
    {
        for (uint32_t i = 0;; ++i)
        {
            blend(row[plane(j) + i], row[3 * S + i]);
            if (a > early || i == uint32_t(S) - 1u)
                return i;
        }
    }
};

/* The colour of one sample and its opacity corrected for the step (the first
 * half of composite_sample); all 0 when the sample has no data, so that
 * whatever its unread voxels map to (an infinite table entry, say) leaves the
 * ray as it is. */
template <int FILTER, bool RAW, class HV>
__device__ __forceinline__ float4 classify_sample(const HV& H, float ac, const Taps<FILTER>& T,
                                                  bool valid)
{
    float4 src = tf_lookup<0>(H, interp<FILTER, RAW>(T));
    const float am = fminf(src.w, 1.0f - 1.0f / 256.0f);
    src.w = 1.0f - ex2_approx(ac * lg2_approx(1.0f - am));
    return valid ? src : make_float4(0.f, 0.f, 0.f, 0.f);
}

constexpr uint32_t kSplitThreads = 64;
constexpr float kRayOver = -3.0e38f; /* RayState::thi of a ray with no sample left */

/* One CTA of kSplitThreads threads per tile of tile_w * tile_h =
 * kSplitThreads / S pixels, S lanes to a ray; block i renders tile order[i]
 * (null: tile i). One sample of look-ahead per lane, as march(). */
template <int DT, int FILTER, int EDGE, int S>
__global__ void __launch_bounds__(kSplitThreads)
    raycast_split_kernel(const RayView V, uint32_t tile_w, uint32_t tile_h,
                         const uint32_t* __restrict__ order)
{
    if (skip_frame(V))
        return;
    /* two rows per ray in turn: by the time a lane writes a row again, every
     * lane has read it, since all have passed the other row's barrier */
    __shared__ alignas(16) float rows[2][kSplitThreads / S * RayGroup<S>::kRow];
    constexpr bool RAW = raw_taps<DT, FILTER, EDGE>();
    const uint32_t n = frame_samples(V);
    const float step = __fdiv_rn(1.0f, __uint2float_rn(n));
    const float ac = __fdiv_rn(32.0f, __uint2float_rn(n));
    const uint32_t tiles_x = (V.W + tile_w - 1) / tile_w;
    const uint32_t tile = order ? order[blockIdx.x] : blockIdx.x;
    const uint32_t ray = threadIdx.x / S, j = threadIdx.x % S;
    const uint32_t px = (tile % tiles_x) * tile_w + ray % tile_w;
    const uint32_t py = (tile / tiles_x) * tile_h + ray / tile_w;
    const bool in = px < V.W && py < V.H;
    RayGeom g;
    g.dir[0] = g.dir[1] = g.dir[2] = g.tg = g.tlo = g.thi = 0.0f;
    g.hit = false;
    float4 init = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in)
    {
        g = ray_setup(V, px, py);
        init = initial_dst(V, px, py);
    }
    RayState r;
    r.tg = r.kf = 0.0f;
    r.kf_safe = -1.0f;
    r.err = 0u;
    r.entry = kLeafEmpty;
    r.brick = nullptr;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        r.dir[a] = r.sa[a] = r.sb[a] = 0.0f;
    if (!ray_begin(g, step, r) || init.w > V.early)
        r.thi = kRayOver;
    r.kf += float(j);
    RayGroup<S> G;
    G.c = (j & 3u) == 0u ? init.x : (j & 3u) == 1u ? init.y : init.z;
    G.a = init.w;
    float* row0 = rows[0] + ray * RayGroup<S>::kRow;
    float* row1 = rows[1] + ray * RayGroup<S>::kRow;
    uint32_t nsamp = 0;
    auto composite = [&](float* row, const Taps<FILTER>& T, bool valid) {
        const float4 src = classify_sample<FILTER, RAW>(V, ac, T, valid);
        row[j] = src.x;
        row[S + j] = src.y;
        row[2 * S + j] = src.z;
        row[3 * S + j] = src.w;
        __syncwarp();
        nsamp += valid ? 1u : 0u;
        if (G.blend_row(row, j, V.early) && r.thi != kRayOver)
        {
            /* the ray ends within this row (once per ray): the samples after
             * the one that passed the opacity do not count */
            const uint32_t last = G.blend_to_stop(row, j, V.early);
            if (valid && j > last)
                --nsamp;
            r.thi = kRayOver;
        }
    };
    Taps<FILTER> T0, T1;
    bool v0, v1;
    bool live = fetch_sample<DT, FILTER, EDGE, S>(V, V, r, step, T0, v0);
    while (__any_sync(0xFFFFFFFFu, live))
    {
        fetch_sample<DT, FILTER, EDGE, S>(V, V, r, step, T1, v1);
        composite(row0, T0, v0);
        v1 = v1 && r.thi != kRayOver;
        live = fetch_sample<DT, FILTER, EDGE, S>(V, V, r, step, T0, v0);
        composite(row1, T1, v1);
        v0 = v0 && r.thi != kRayOver;
    }
    flush_error(V, r);
    if (in && j < 4u)
        reinterpret_cast<float*>(V.out + frame_index(V, px, py))[j] = j == 3u ? G.a : G.c;
    unsigned long long sum = nsamp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31u) == 0 && sum)
        atomicAdd(reinterpret_cast<unsigned long long*>(V.counters + FC_SAMPLES_LO), sum);
}

template <int DT, int FILTER, int EDGE>
TileKernel split_kernel_of(uint32_t lanes)
{
    return lanes == 4 ? raycast_split_kernel<DT, FILTER, EDGE, 4>
                      : raycast_split_kernel<DT, FILTER, EDGE, 8>;
}

} // namespace
} // namespace lv
