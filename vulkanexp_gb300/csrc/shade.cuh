// shade.cuh — hit shading of a probe ray: sampleProbes (the infinite-bounce
// lookup into the previous atlas), the sun BRDF, and the closest-hit program
// of the reference with NO_REFLECTION.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace ddgi {

// Atlas views.  FP32 form: float4 colour (RGBA) and float2 depth texels;
// FP16 form: 4 x half colour and 2 x half depth texels.
struct ColorTexF32 {
    static constexpr uint32_t kBytes = 16;
    const float4* p;
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        float4 v = __ldg(p + i);
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
    }
};
struct DepthTexF32 {
    static constexpr uint32_t kBytes = 8;
    const float2* p;
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        float2 v = __ldg(p + i);
        o[0] = v.x;
        o[1] = v.y;
    }
};
struct ColorTexF16 {
    static constexpr uint32_t kBytes = 8;
    const uint2* p;  // 4 halves
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        uint2 v = __ldg(p + i);
        __half2 a = *reinterpret_cast<__half2*>(&v.x);
        __half2 b = *reinterpret_cast<__half2*>(&v.y);
        float2 fa = __half22float2(a), fb = __half22float2(b);
        o[0] = fa.x;
        o[1] = fa.y;
        o[2] = fb.x;
    }
};
struct DepthTexF16 {
    static constexpr uint32_t kBytes = 4;
    const uint32_t* p;  // 2 halves
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        uint32_t v = __ldg(p + i);
        float2 f = __half22float2(*reinterpret_cast<__half2*>(&v));
        o[0] = f.x;
        o[1] = f.y;
    }
};

// Either form, chosen per lookup at run time (the batched kernels, whose
// volumes may mix the forms): one copy of the shading code instead of one
// per form.
struct ColorTexDyn {
    const void* p;
    bool half;
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        if (half) ColorTexF16{static_cast<const uint2*>(p)}.fetch(i, o);
        else ColorTexF32{static_cast<const float4*>(p)}.fetch(i, o);
    }
};
struct DepthTexDyn {
    const void* p;
    bool half;
    __device__ __forceinline__ void fetch(size_t i, float* o) const {
        if (half) DepthTexF16{static_cast<const uint32_t*>(p)}.fetch(i, o);
        else DepthTexF32{static_cast<const float2*>(p)}.fetch(i, o);
    }
};

template <class CT, class DT>
struct AtlasView {
    CT color;
    DT depth;
};

// The lookup's arithmetic is written with explicit fmaf / __fmul_rn where a
// product meets a sum, so that every kernel it is inlined into (single and
// batched, FP32 and FP16 atlas) rounds alike.
__device__ __forceinline__ float dot_fma(float3 a, float3 b) {
    return fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x)));
}
// The products and sums of a hit's surface and of its sun term, each rounded in
// one way in every kernel that shades hits.
__device__ __forceinline__ float mix_of_three(float x, float a, float y, float b, float z, float c) {
    return fmaf(z, c, fmaf(x, a, __fmul_rn(y, b)));
}
__device__ __forceinline__ float dot_hit(float3 a, float3 b) { return mix_of_three(a.x, b.x, a.y, b.y, a.z, b.z); }
__device__ __forceinline__ float3 norm_hit(float3 a) {
    const float k = 1.0f / sqrtf(dot_hit(a, a));
    return f3(__fmul_rn(a.x, k), __fmul_rn(a.y, k), __fmul_rn(a.z, k));
}
__device__ __forceinline__ float sqrt_approx(float v) {  // within 2^-23 relative (PTX sqrt.approx)
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// The same of three radiances.  The form that takes subnormal numbers costs
// three instructions more a root, which the 24 roots of a lookup would feel (a
// 1920x1080 final gather 91 us against 87), so it is kept for them.
__device__ __forceinline__ void sqrt_approx3(const float (&v)[3], float (&r)[3]) {
    if (fmin3(v[0], v[1], v[2]) < 0x1p-126f) {
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = sqrt_approx(v[k]);
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r[k]) : "f"(v[k]));
    }
}

// Octahedral coordinates of a direction of length one (irradiance.glsl:119-138)
// with one reciprocal for its quotients.  Each quotient is brought to the
// correctly rounded one by its remainder (Markstein 1990: q + (a - q b) / b
// with the reciprocal refined by a Newton step), so the mapping has the bits
// of a division (below 2^-102 a quotient can differ, which the added half
// hides): next to a probe of strong contrast one unit in the last place of uv
// shows in the result's sixth digit.
__device__ __forceinline__ float2 oct_uv(float3 d) {
    const float sum = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    float r = __fdividef(1.0f, sum);
    r = fmaf(r, fmaf(-sum, r, 1.0f), r);
    float x = __fmul_rn(d.x, r), y = __fmul_rn(d.y, r);
    x = fmaf(fmaf(-sum, x, d.x), r, x);
    y = fmaf(fmaf(-sum, y, d.y), r, y);
    if (d.z < 0.0f) {  // fold; like the reference's sign(), 0 folds to 0
        const float fx = d.x != 0.0f ? copysignf(1.0f - fabsf(y), d.x) : 0.0f;
        const float fy = d.y != 0.0f ? copysignf(1.0f - fabsf(x), d.y) : 0.0f;
        x = fx;
        y = fy;
    }
    return make_float2(fmaf(x, 0.5f, 0.5f), fmaf(y, 0.5f, 0.5f));
}

// The four texels of a lookup and their bilinear weights.  The reference's
// coordinate is ((side tile + 1) / side + (side - 2) / side uv) / tiles, and
// the texel position that times the atlas width, side x tiles, less half a
// texel.  Here the quotient by `tiles` and its product are left out (exact
// inverses of each other on grids of powers of two, one rounding less on the
// others); the sum of tile and uv is rounded as the reference's, so for sides
// that are powers of two the fraction has the reference's bits (for others
// 1 / side is rounded before the sum).  A lookup stays at least half a texel
// inside its tile; the clamps keep a NaN's in the atlas too.
struct Tap {
    uint32_t row0, row1;  // first texel in the upper and in the lower row
    float ax, ay;
};
// tx, ty: tile + 1 / side along the axes; scale: (side - 2) / side
__device__ __forceinline__ Tap atlas_tap(float tx, float ty, float2 uv, float scale, float side, uint32_t w, uint32_t h) {
    const float x = fmaf(fmaf(scale, uv.x, tx), side, -0.5f), y = fmaf(fmaf(scale, uv.y, ty), side, -0.5f);
    const float x0 = floorf(x), y0 = floorf(y);
    Tap t;
    t.ax = x - x0;
    t.ay = y - y0;
    const int i = min(max((int)x0, 0), (int)w - 2), j = min(max((int)y0, 0), (int)h - 2);
    t.row0 = (uint32_t)j * w + (uint32_t)i;
    t.row1 = t.row0 + w;
    return t;
}

// Scales of one lookup's coordinates and of its eight probes.
struct LookupScales {
    float cr, dr, cscale, dscale, cinv, dinv;
};
__device__ __forceinline__ LookupScales lookup_scales(const DeviceGrid& g) {
    LookupScales s;
    s.cr = (float)g.color_res;
    s.dr = (float)g.depth_res;
    s.cscale = (float)(g.color_res - 2) / s.cr;
    s.dscale = (float)(g.depth_res - 2) / s.dr;
    s.cinv = 1.0f / s.cr;
    s.dinv = 1.0f / s.dr;
    return s;
}

// The eight probes around a position: its cell (as exact floats), and which
// of the cell's corners are on the grid and not OFF.
struct ProbeCell {
    float x, y, z;
    uint32_t live;  // bit i: corner i (offsets along x, y, z in bits 0, 1, 2) counts
};
// false: outside the grid's lower bounds (or NaN), where a lookup returns 0.
__device__ __forceinline__ bool probe_cell(float3 position, const DeviceGrid& g, const uint32_t* states, ProbeCell* c) {
    const float3 at = (position - f3(g.mn[0], g.mn[1], g.mn[2])) / f3(g.cell[0], g.cell[1], g.cell[2]);
    if (!(at.x >= 0.0f && at.y >= 0.0f && at.z >= 0.0f)) return false;
    // the clamp only matters beyond 2^24 cells, where every corner is off-grid
    c->x = floorf(fminf(at.x, 16777216.0f));
    c->y = floorf(fminf(at.y, 16777216.0f));
    c->z = floorf(fminf(at.z, 16777216.0f));
    const int x = (int)c->x, y = (int)c->y, z = (int)c->z;
    const uint32_t sx = (uint32_t)g.res[0], sxy = sx * (uint32_t)g.res[1];
    const uint32_t lin = (uint32_t)x + sx * (uint32_t)y + sxy * (uint32_t)z;
    c->live = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // eight loads in flight at once
        const int ox = i & 1, oy = (i >> 1) & 1, oz = i >> 2;
        if (x + ox < g.res[0] && y + oy < g.res[1] && z + oz < g.res[2] &&
            __ldg(states + lin + ox + (oy ? sx : 0u) + (oz ? sxy : 0u)) != 0u)
            c->live |= 1u << i;
    }
    return true;
}

// One corner of the cell: its position, the way to it from the lookup's
// position, 1 / its length, its trilinear weight, and its tile along the
// atlas axes (x + res.x y and z; exact: a grid has at most 2^24 probes).
struct CellProbe {
    float3 at, v;
    float inv_len, triw, tile, z;
};
__device__ __forceinline__ CellProbe cell_probe(const ProbeCell& c, uint32_t i, float3 position, const DeviceGrid& g) {
    const float x = c.x + ((i & 1u) ? 1.0f : 0.0f), y = c.y + ((i & 2u) ? 1.0f : 0.0f);
    CellProbe p;
    p.z = c.z + ((i & 4u) ? 1.0f : 0.0f);
    p.tile = fmaf(y, (float)g.res[0], x);
    p.at = f3(fmaf(x, g.cell[0], g.mn[0]), fmaf(y, g.cell[1], g.mn[1]), fmaf(p.z, g.cell[2], g.mn[2]));
    p.v = p.at - position;
    p.triw = fmaf(__fmul_rn(__saturatef(fmaf(-fabsf(p.v.x), g.inv_cell[0], 1.0f)),
                            __saturatef(fmaf(-fabsf(p.v.y), g.inv_cell[1], 1.0f))),
                  __saturatef(fmaf(-fabsf(p.v.z), g.inv_cell[2], 1.0f)), 0.001f);
    p.inv_len = rsqrtf(dot_fma(p.v, p.v));
    return p;
}

// Facing and Chebyshev visibility (irradiance.glsl:188-222) of probe p for
// one lookup, `bv` the way to it from the biased position: the weight and the
// weight without visibility.
template <class DT>
__device__ __forceinline__ void probe_weights(const CellProbe& p, float3 bv, float3 normal, const DT& tex,
                                              const LookupScales& s, const DeviceGrid& g, float* weight,
                                              float* fallback) {
    const float d2 = dot_fma(bv, bv);
    const float2 uv = oct_uv(bv * -rsqrtf(d2));  // the direction from the probe, of length 1 as in the reference
    const Tap t = atlas_tap(p.tile + s.dinv, p.z + s.dinv, uv, s.dscale, s.dr, g.depth_w, g.depth_h);
    float a[2], b[2], c[2], d[2], m[2];
    tex.fetch(t.row0, a);
    tex.fetch(t.row0 + 1u, b);
    tex.fetch(t.row1, c);
    tex.fetch(t.row1 + 1u, d);
    const float facing = fmaxf(0.0001f, fmaf(__fmul_rn(dot_fma(p.v, normal), p.inv_len), 0.5f, 0.5f));
    float w = fmaf(facing, facing, 0.2f);
    *fallback = __fmul_rn(w, p.triw);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float top = fmaf(t.ax, b[k] - a[k], a[k]), bot = fmaf(t.ax, d[k] - c[k], c[k]);
        m[k] = fmaf(t.ay, bot - top, top);
    }
    const float dist = sqrt_approx(d2);
    const float variance = fabsf(fmaf(m[0], m[0], -m[1]));
    // the quotient of a sixteenth of either side, which has the same bits: the
    // approximate division gives 0 for a divisor above 2^126
    const float dm = __fmul_rn(fmaxf(dist - m[0], 0.0001f), 0.25f), part = __fmul_rn(variance, 0.0625f);
    const float cheb = __fdividef(part, fmaf(dm, dm, part));
    w = __fmul_rn(w, (dist <= m[0]) ? 1.0f : fmaxf(__fmul_rn(__fmul_rn(cheb, cheb), cheb), 0.0f));
    w = fmaxf(0.000001f, w);
    const float crush = 0.2f;
    if (w < crush) w = __fmul_rn(w, __fmul_rn(__fmul_rn(w, w), 1.0f / (crush * crush)));
    *weight = __fmul_rn(w, p.triw);
}

// The biased position itself is rounded, as in the reference: where the
// distance from it is the stored mean distance, visibility jumps.
__device__ __forceinline__ float3 biased_position(float3 position, float3 normal, float3 toCamera,
                                                  const DeviceGrid& g) {
    return f3(fmaf(normal.x + toCamera.x, g.bias, position.x), fmaf(normal.y + toCamera.y, g.bias, position.y),
              fmaf(normal.z + toCamera.z, g.bias, position.z));
}

// What probe p gives to one lookup: its irradiance's square root, its weight
// and its weight without visibility.
struct ProbeShare {
    float r[3];
    float weight, fallback;
};
template <class AV>
__device__ __forceinline__ ProbeShare probe_share(const CellProbe& p, float3 biasedPosition, float3 normal, float2 nuv,
                                                  const LookupScales& s, const DeviceGrid& g, const AV& at) {
    const Tap t = atlas_tap(p.tile + s.cinv, p.z + s.cinv, nuv, s.cscale, s.cr, g.color_w, g.color_h);
    float c00[3], c10[3], c01[3], c11[3];
    at.color.fetch(t.row0, c00);
    at.color.fetch(t.row0 + 1u, c10);
    at.color.fetch(t.row1, c01);
    at.color.fetch(t.row1 + 1u, c11);
    ProbeShare x;
    probe_weights(p, p.at - biasedPosition, normal, at.depth, s, g, &x.weight, &x.fallback);
    const float w11 = __fmul_rn(t.ax, t.ay), w10 = t.ax - w11, w01 = t.ay - w11, w00 = 1.0f - t.ax - w01;
    float c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = fmaf(w11, c11[k], fmaf(w01, c01[k], fmaf(w10, c10[k], __fmul_rn(w00, c00[k]))));
    sqrt_approx3(c, x.r);
    return x;
}

// The probes' shares of one lookup added up in their order.
struct LookupSum {
    float final[3] = {0.0f, 0.0f, 0.0f}, other[3] = {0.0f, 0.0f, 0.0f};
    float weight = 0.0f, fallback = 0.0f;

    __device__ __forceinline__ void add(const ProbeShare& x) {
#pragma unroll
        for (int k = 0; k < 3; ++k) final[k] = fmaf(x.r[k], x.weight, final[k]);
        weight += x.weight;
#pragma unroll
        for (int k = 0; k < 3; ++k) other[k] = fmaf(x.r[k], x.fallback, other[k]);
        fallback += x.fallback;
    }
    __device__ __forceinline__ float3 color() const {
        const float n = weight > 1e-3f ? 1.0f / weight : 1.0f;
        const float nf = fallback > 1e-3f ? 1.0f / fallback : 1.0f;
        const float k = 8.0f * clampf(weight, 0.0f, 1.0f / 8.0f);
        float r[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float fc = __fmul_rn(final[c], n), fb = __fmul_rn(other[c], nf);
            r[c] = fmaf(__fmul_rn(fb, fb), 1.0f - k, __fmul_rn(__fmul_rn(fc, fc), k));
        }
        return f3(r[0], r[1], r[2]);
    }
};

// sampleProbes (src/shaders/irradiance.glsl:145-237) for NQ lookups at one
// position that differ in the direction argument (`normal`): the closest-hit
// program makes two (reflection and diffuse), which share the eight probes'
// states, positions, directions and trilinear weights.
//
// Bound by instruction issue where many lookups run (the final gather, a
// large update's shading) and by the chain of loads where few do.  So the
// coordinates are formed without the quotient and product by the atlas size,
// square roots and the visibility quotient are the approximate instructions
// (2 ulp, far below the cancellation in the variance), and the eight states
// are loaded together.  Against the
// reference's expressions as written: a 1920x1080 final gather over a 16-bit
// atlas 141 -> 87 us (1,980 warp instructions a warp before), 643x361 over an
// FP32 atlas 50 -> 37 us, the shading of 65 K hits 39 -> 24 us and of an
// update's 2.6 M 518 -> 375 us.  Distance from a 64-bit evaluation, root mean
// square of six gathers over 16- and 32-bit atlases: 4.0e-7, 4.8e-7, 5.5e-7,
// 6.7e-7, 1.1e-6 and 1.3e-5 (a probe's visibility jumping), before 4.0e-7,
// 4.9e-7, 5.5e-7, 8.2e-7, 1.2e-6 and 1.3e-5.  With correctly rounded roots and
// quotients it is the same to three digits and the 1920x1080 gather 112 us.
template <int NQ, class AV>
__device__ void sample_probes_n(float3 position, const float3 (&normal)[NQ], float3 toCamera, const DeviceGrid& g,
                                const uint32_t* states, const AV& at, float3 (&result)[NQ]) {
    ProbeCell cell;
#pragma unroll
    for (int q = 0; q < NQ; ++q) result[q] = f3(0, 0, 0);
    if (!probe_cell(position, g, states, &cell)) return;
    const LookupScales s = lookup_scales(g);
    float3 biasedPosition[NQ];
    float2 nuv[NQ];
    LookupSum sum[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        biasedPosition[q] = biased_position(position, normal[q], toCamera, g);
        nuv[q] = oct_uv(normal[q]);
    }
#pragma unroll 1
    for (uint32_t live = cell.live; live != 0u; live &= live - 1u) {
        const CellProbe p = cell_probe(cell, (uint32_t)__ffs((int)live) - 1u, position, g);
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            sum[q].add(probe_share(p, biasedPosition[q], normal[q], nuv[q], s, g, at));
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) result[q] = sum[q].color();
}

// One lookup by PARTS neighbouring lanes of a warp, all of which call it (those
// without a lookup with `valid` false): each takes every PARTS-th of the eight
// probes, and all add the shares up in the probes' order, so that the sums are
// sample_probes_n's bit for bit.
template <int PARTS, class AV>
__device__ __forceinline__ float3 sample_probes_split(bool valid, float3 position, float3 normal, float3 toCamera,
                                                      const DeviceGrid& g, const uint32_t* states, const AV& at) {
    ProbeCell cell;
    if (!valid || !probe_cell(position, g, states, &cell)) cell.live = 0u;
    const uint32_t lane = threadIdx.x & 31u, part = lane % PARTS, lead = lane - part;
    const LookupScales s = lookup_scales(g);
    const float3 biased = biased_position(position, normal, toCamera, g);
    const float2 nuv = oct_uv(normal);
    LookupSum sum;
#pragma unroll 1
    for (uint32_t j = 0; j < 8u; j += PARTS) {
        ProbeShare own = {{0.0f, 0.0f, 0.0f}, 0.0f, 0.0f};  // a share of nothing changes no sum
        if (cell.live >> (j + part) & 1u)
            own = probe_share(cell_probe(cell, j + part, position, g), biased, normal, nuv, s, g, at);
#pragma unroll
        for (uint32_t p = 0; p < (uint32_t)PARTS; ++p) {
            ProbeShare x = own;
            if (PARTS > 1) {
#pragma unroll
                for (int k = 0; k < 3; ++k) x.r[k] = __shfl_sync(0xffffffffu, own.r[k], lead + p);
                x.weight = __shfl_sync(0xffffffffu, own.weight, lead + p);
                x.fallback = __shfl_sync(0xffffffffu, own.fallback, lead + p);
            }
            sum.add(x);
        }
    }
    return sum.color();
}

template <class AV>
__device__ __forceinline__ float3 sample_probes(float3 position, float3 normal, float3 toCamera, const DeviceGrid& g,
                                                const uint32_t* states, const AV& at) {
    const float3 n[1] = {normal};
    float3 r[1];
    sample_probes_n<1>(position, n, toCamera, g, states, at, r);
    return r[0];
}

// pbrMetallicRoughness (src/shaders/pbrMetallicRoughness.glsl:43-84)
__device__ __forceinline__ float3 pbr_metallic_roughness(float3 n, float3 v, float3 lightColor, float3 lightDir,
                                                         float3 albedo, float metal, float rough) {
    const float pi = DDGI_PI;
    const float alphaRoughness = __fmul_rn(rough, rough), dull = 1.0f - metal;
    const float al[3] = {albedo.x, albedo.y, albedo.z}, lc[3] = {lightColor.x, lightColor.y, lightColor.z};
    float R0[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) R0[c] = fmaf(0.04f, dull, __fmul_rn(al[c], metal));
    const float reflectance = fmaxf(fmaxf(R0[0], R0[1]), R0[2]);
    const float R90 = clampf(__fmul_rn(reflectance, 25.0f), 0.0f, 1.0f);
    const float3 l = norm_hit(lightDir);
    const float3 h = norm_hit(l + v);
    const float NdotL = clampf(dot_hit(n, l), 0.001f, 1.0f);
    const float NdotV = clampf(fabsf(dot_hit(n, v)), 0.001f, 1.0f);
    const float NdotH = clampf(dot_hit(n, h), 0.0f, 1.0f);
    const float VdotH = clampf(dot_hit(v, h), 0.0f, 1.0f);
    const float x = clampf(1.0f - VdotH, 0.0f, 1.0f);
    const float x2 = __fmul_rn(x, x);
    const float p5 = __fmul_rn(__fmul_rn(x2, x2), x);
    const float rest = fmaf(-alphaRoughness, alphaRoughness, 1.0f);
    const float attL = __fmul_rn(2.0f, NdotL) /
                       (NdotL + sqrtf(fmaf(alphaRoughness, alphaRoughness, __fmul_rn(rest, __fmul_rn(NdotL, NdotL)))));
    const float attV = __fmul_rn(2.0f, NdotV) /
                       (NdotV + sqrtf(fmaf(alphaRoughness, alphaRoughness, __fmul_rn(rest, __fmul_rn(NdotV, NdotV)))));
    const float a = __fmul_rn(NdotH, alphaRoughness);
    const float k = alphaRoughness / fmaf(a, a, fmaf(-NdotH, NdotH, 1.0f));
    const float D = clampf(__fmul_rn(__fmul_rn(k, k), 1.0f / pi), 0.0f, 4.0f);
    const float spec = __fmul_rn(__fmul_rn(attL, attV), D) / __fmul_rn(__fmul_rn(4.0f, NdotL), NdotV);
    float out[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float F = fmaf(R90 - R0[c], p5, R0[c]);
        const float diffuse = __fmul_rn(__fmul_rn(al[c], 1.0f - 0.04f), dull);
        const float both = fmaf(__fmul_rn(1.0f - F, diffuse), 1.0f / pi, __fmul_rn(F, spec));
        out[c] = __fmul_rn(__fmul_rn(lc[c], both), NdotL);
    }
    return f3(out[0], out[1], out[2]);
}

// Front-face hit shading of src/shaders/closesthit.glsl:143-286 (NO_REFLECTION,
// no textures), split around the shadow query: `base` is emissive + specular
// bounce + diffuse bounce, `sun` the unshadowed sun term and `fade` the
// night fade (1 when the sun is above the horizon).  The shaded colour is
// base if the shadow ray hits, else (base + sun) * fade, which is the
// reference's `color += pbr; if (dir.y < 0) color *= fade`.
struct SurfaceShade {
    float3 base, sun, position;
    float fade;
};

// Geometry and material at a front-face hit (closesthit.glsl:143-190, no
// textures).
struct Surface {
    float3 position, normal, albedo, emissive;
    float metal, rough;
    uint32_t material;
};

__device__ __forceinline__ bool surface_at(const DeviceScene& sc, float3 origin, float3 dir, float t, float b1,
                                           float b2, uint32_t inst, uint32_t prim, Surface* s, uint32_t* err) {
    // hit position: product then sum, each rounded (shared with the shadow ray)
    s->position = f3(__fadd_rn(__fmul_rn(dir.x, t), origin.x), __fadd_rn(__fmul_rn(dir.y, t), origin.y),
                     __fadd_rn(__fmul_rn(dir.z, t), origin.z));
    const GpuInstance* gi = sc.instances_by_id + inst;
    uint32_t custom = __ldg(&gi->custom);
    ddgi_offset_entry oe = sc.offsets[custom];
    uint32_t io = oe.index_offset + 3u * prim;
    uint32_t i0 = __ldg(sc.indices + io), i1 = __ldg(sc.indices + io + 1), i2 = __ldg(sc.indices + io + 2);
    uint32_t vb = oe.vertex_offset;
    if (vb + max(i0, max(i1, i2)) >= sc.vertex_count || oe.material_index >= sc.material_count) {
        raise_error(err, DEV_BAD_INDEX);
        return false;
    }
    float4 n0 = __ldg(sc.normals + vb + i0), n1 = __ldg(sc.normals + vb + i1), n2 = __ldg(sc.normals + vb + i2);
    float b0 = 1.0f - b1 - b2;
    float3 tsn = norm_hit(f3(mix_of_three(n0.x, b0, n1.x, b1, n2.x, b2), mix_of_three(n0.y, b0, n1.y, b1, n2.y, b2),
                             mix_of_three(n0.z, b0, n1.z, b1, n2.z, b2)));
    float4 w0 = __ldg(&gi->w2o[0]), w1 = __ldg(&gi->w2o[1]), w2 = __ldg(&gi->w2o[2]);
    // normal * gl_WorldToObjectEXT: transpose of the world-to-object 3x3
    s->normal = norm_hit(f3(mix_of_three(tsn.x, w0.x, tsn.y, w1.x, tsn.z, w2.x),
                            mix_of_three(tsn.x, w0.y, tsn.y, w1.y, tsn.z, w2.y),
                            mix_of_three(tsn.x, w0.z, tsn.y, w1.z, tsn.z, w2.z)));
    const ddgi_material& m = sc.materials[oe.material_index];
    s->albedo = f3(m.base_color[0], m.base_color[1], m.base_color[2]);
    s->emissive = f3(m.emissive[0], m.emissive[1], m.emissive[2]);
    s->metal = m.metallic;
    s->rough = m.roughness;
    s->material = oe.material_index;
    return true;
}

__device__ __forceinline__ float3 reflected(float3 dir, float3 normal) {
    const float k = -2.0f * dot_hit(normal, dir);
    return f3(fmaf(normal.x, k, dir.x), fmaf(normal.y, k, dir.y), fmaf(normal.z, k, dir.z));
}

// The shading of surface `s` seen along `dir` from the two lookups' results.
// Written with explicit multiply-adds here and in the lookups: several kernels
// shade hits, and all give the same bits.
__device__ __forceinline__ void shade_from_lookups(const Surface& s, const DeviceLight& L, float3 dir,
                                                   float3 reflection, float3 indirect, SurfaceShade* out) {
    out->position = s.position;
    const float3 normal = s.normal, albedo = s.albedo;
    const float metal = s.metal, rough = s.rough;
    const float a[3] = {albedo.x, albedo.y, albedo.z}, r[3] = {reflection.x, reflection.y, reflection.z},
                i[3] = {indirect.x, indirect.y, indirect.z};
    float color[3] = {s.emissive.x, s.emissive.y, s.emissive.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float diffuse = __fmul_rn(__fmul_rn(a[c], 1.0f - 0.04f), 1.0f - metal);
        const float specular = fmaf(0.04f, 1.0f - metal, __fmul_rn(a[c], metal));
        color[c] = fmaf(i[c], diffuse, fmaf(specular, r[c], color[c]));
    }
    out->base = f3(color[0], color[1], color[2]);
    out->sun = pbr_metallic_roughness(normal, norm_hit(-dir), f3(L.color[0], L.color[1], L.color[2]),
                                      f3(L.dir[0], L.dir[1], L.dir[2]), albedo, metal, rough);
    out->fade = L.dir[1] < 0.0f ? 1.0f - clampf(-L.dir[1], 0.0f, 0.1f) / 0.1f : 1.0f;
}
// What a hit whose indices are out of range shades to.
__device__ __forceinline__ void shade_nothing(float3 position, SurfaceShade* out) {
    out->position = position;
    out->base = out->sun = f3(0, 0, 0);
    out->fade = 1.0f;
}

template <class AV>
__device__ __forceinline__ bool shade_surface(const DeviceScene& sc, const DeviceGrid& g, const DeviceLight& L,
                                              const uint32_t* states, const AV& at, float3 origin, float3 dir,
                                              float t, float b1, float b2, uint32_t inst, uint32_t prim,
                                              SurfaceShade* out, uint32_t* err) {
    Surface s;
    if (!surface_at(sc, origin, dir, t, b1, b2, inst, prim, &s, err)) {
        shade_nothing(s.position, out);
        return false;
    }
    const float3 lookups[2] = {reflected(dir, s.normal), s.normal};
    float3 sampled[2];  // reflection, indirect
    sample_probes_n<2>(s.position, lookups, -dir, g, states, at, sampled);
    shade_from_lookups(s, L, dir, sampled[0], sampled[1], out);
    return true;
}

__device__ __forceinline__ float3 lit_color(const SurfaceShade& s) { return (s.base + s.sun) * s.fade; }

}  // namespace ddgi
