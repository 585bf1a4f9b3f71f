// adjoint.cu — reverse-mode gradients of a colour-atlas loss through K
// recurrent probe updates, with the hit set held fixed.
//
// Forward of one update k (FP32 form, all probes), for a probe ray:
//   miss:      x = sky
//   backface:  x = 0
//   front hit: base = emissive + spec(albedo) * sampleProbes_k-1(reflect)
//                              + diffuse(albedo) * sampleProbes_k-1(normal)
//              x = shadowed ? base : (base + pbr(albedo) * sun) * fade
// and the colour blend of every interior texel t of the probe:
//   atlas_k[t] = (1 - h) * sum_r w[t][r] x_r / W_t + h * atlas_k-1[t]
// followed by the border copy.  The depth atlas does not depend on albedo,
// sun or sky once the hits are fixed, so only the colour chain is reversed.
//
// Reverse step k, given G_k = dL/d atlas_k:
//   k_blend_adjoint   border gradients go to their source interior texels,
//                     G_k-1 (interior) = h G_k, g_x[r] = (1-h) sum_t w W^-1 G;
//   k_ray_adjoint     g_x -> albedo, sun and sky gradients, and the two
//                     sampleProbes lookups scatter into G_k-1 (atomics).
// atlas_k-1 itself is restored from a checkpoint and replayed (k_replay_shade
// + the FP32 blend), so no hit is traced again.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "shade.cuh"

namespace ddgi {

namespace {

using AtlasF32 = AtlasView<ColorTexF32, DepthTexF32>;
constexpr uint32_t kShadowBit = 1u << 30;
constexpr uint32_t kBackBit = 1u << 31;
constexpr uint32_t kPrimMask = (1u << 28) - 1u;

__device__ __forceinline__ float night_fade(const DeviceLight& L) {
    return L.dir[1] < 0.0f ? 1.0f - clampf(-L.dir[1], 0.0f, 0.1f) / 0.1f : 1.0f;
}

// One ray record from a recorded hit (the forward's shading, no traversal).
__global__ void __launch_bounds__(128) k_replay_shade(DeviceScene sc, DeviceGrid g, DeviceLight L,
                                                      const float4* __restrict__ dirs,
                                                      const uint32_t* __restrict__ states, AtlasF32 at,
                                                      const float4* __restrict__ thit,
                                                      const uint32_t* __restrict__ prim, float4* rays, uint32_t total,
                                                      uint32_t* err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const uint32_t R = g.rays, slot = i / R, ray = i - slot * R;
    float4 th = thit[i];
    uint32_t pb = prim[i], inst = __float_as_uint(th.w);
    float4 rec;
    if (inst == 0xFFFFFFFFu) {
        rec = make_float4(L.sky[0], L.sky[1], L.sky[2], -1.0f);
    } else if (pb & kBackBit) {
        rec = make_float4(0.0f, 0.0f, 0.0f, th.x * 0.80f);
    } else {
        float4 d4 = dirs[ray];
        SurfaceShade s;
        shade_surface(sc, g, L, states, at, probe_origin_exact(g, slot), f3(d4.x, d4.y, d4.z), th.x, th.y, th.z, inst,
                      pb & kPrimMask, &s, err);
        float3 c = (pb & kShadowBit) ? s.base : lit_color(s);
        rec = make_float4(c.x, c.y, c.z, th.x);
    }
    rays[i] = rec;
}

// Gradient of an interior texel (sx, sy) of the tile at (ox, oy): its own and
// those of the border texels that copy it (the inverse of border_entry).
__device__ __forceinline__ float3 folded_gradient(const float4* __restrict__ g, size_t ox, size_t oy, uint32_t w, int n,
                                                  int sx, int sy) {
    const int e = n - 1, m = n - 2;
    float3 s = f3(0, 0, 0);
    auto take = [&](bool copied, int x, int y) {
        if (!copied) return;
        const float4 v = __ldg(g + (oy + y) * w + ox + x);
        s = s + f3(v.x, v.y, v.z);
    };
    take(true, sx, sy);
    take(sx == 1, 0, e - sy);
    take(sx == m, e, e - sy);
    take(sy == 1, e - sx, 0);
    take(sy == m, e - sx, e);
    take(sx == m && sy == m, 0, 0);
    take(sx == m && sy == 1, 0, e);
    take(sx == 1 && sy == m, e, 0);
    take(sx == 1 && sy == 1, e, e);
    return s;
}

// Adjoint of the colour blend + hysteresis + border copy of one probe (block =
// probe).  wsum: the colour texels' weight sums, as the forward adds them up
// (one launch for all probes; each block adding up its own, a chain of 256
// loads by 36 threads, took 43 us for 2,048 probes of 256 rays, and a pass of
// its own for the border 14 us; 17 us now and 7 us for the sums).
__global__ void __launch_bounds__(256) k_blend_adjoint(DeviceGrid g, const float4* __restrict__ dirs,
                                                       const float* __restrict__ wsum, const float4* __restrict__ gk,
                                                       float4* gprev, float4* gx) {
    extern __shared__ float smem[];
    const uint32_t R = g.rays;
    const int n = (int)g.color_res - 2, nt = n * n;
    float* s_td = smem;            // nt x 3
    float* s_g = s_td + 3 * nt;    // nt x 3, already divided by W_t
    const uint32_t probe = blockIdx.x;
    const uint32_t rx = (uint32_t)g.res[0], rxy = (uint32_t)(g.res[0] * g.res[1]);
    const int ix = (int)(probe % rx), iy = (int)((probe % rxy) / rx), iz = (int)(probe / rxy);
    const int cres = (int)g.color_res, tile = iy * g.res[0] + ix;
    const size_t ox = (size_t)cres * tile, oy = (size_t)cres * iz;
    const float hy = g.hyst;
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
        int tx = t % n, ty = t / n;
        float sc = texel_scale((uint32_t)n), ce = 0.5f * (float)(n - 1);
        float3 td = oct_decode(sc * ((float)tx - ce), sc * ((float)ty - ce));
        const float W = wsum[t];
        float inv = W > 1e-3f ? 1.0f / W : 1.0f;
        size_t ti = (oy + 1 + ty) * g.color_w + ox + 1 + tx;
        const float3 gv = folded_gradient(gk, ox, oy, g.color_w, cres, 1 + tx, 1 + ty);
        gprev[ti] = make_float4(hy * gv.x, hy * gv.y, hy * gv.z, 0.0f);
        s_td[3 * t] = td.x;
        s_td[3 * t + 1] = td.y;
        s_td[3 * t + 2] = td.z;
        s_g[3 * t] = (1.0f - hy) * gv.x * inv;
        s_g[3 * t + 1] = (1.0f - hy) * gv.y * inv;
        s_g[3 * t + 2] = (1.0f - hy) * gv.z * inv;
    }
    const int nb = 4 + 4 * (cres - 2);
    for (int e = threadIdx.x; e < nb; e += blockDim.x) {
        int4 b = border_entry(e, cres);
        gprev[(oy + b.y) * g.color_w + ox + b.x] = make_float4(0, 0, 0, 0);
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < R; r += blockDim.x) {
        float4 d = dirs[r];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        for (int t = 0; t < nt; ++t) {
            float w = fmaxf(0.0f, s_td[3 * t] * d.x + s_td[3 * t + 1] * d.y + s_td[3 * t + 2] * d.z);
            a0 += w * s_g[3 * t];
            a1 += w * s_g[3 * t + 1];
            a2 += w * s_g[3 * t + 2];
        }
        gx[(size_t)probe * R + r] = make_float4(a0, a1, a2, 0.0f);
    }
}

// Adds (x, y, z, 0) to a texel's gradient: one 16-byte reduction.
__device__ __forceinline__ void add_texel(float4* p, float x, float y, float z) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :
                 : "l"(p), "f"(x), "f"(y), "f"(z), "f"(0.0f)
                 : "memory");
}

constexpr int kAdjointThreads = 128;
constexpr int kLookupWords = 32;  // weights of two lookups' eight probes, per thread in shared memory

// The two lookups of a hit (sampleProbes, irradiance.glsl:145-237) evaluated
// and differentiated with respect to the colour atlas: returns the values,
// and adds d(value)/d(texel) . gout into gatlas.  The weights depend only on
// geometry and the depth atlas (constants here); d sqrt(c)/dc at c = 0 is
// taken as 0 (such texels receive only zero radiance whatever the parameters).
//
// The first pass over the eight probes has the forward's directions and weights
// bit for bit (its colours differ in rounding: their roots are divided by, and
// correctly rounded) and keeps the weights (`w`: this thread's column of
// kLookupWords in shared memory); the second fetches the colours again and
// scatters.  Bound by the L2's reductions, 64 a
// hit: of four floats each, where single floats took 192.  524 K rays of a
// room: 580 us with both passes over everything, a lookup at a time, and
// single-float reductions; 247 us now.
__device__ __forceinline__ void sample_probes_vjp2(float3 position, const float3 (&normal)[2], float3 toCamera,
                                                   const DeviceGrid& g, const uint32_t* states, const AtlasF32& at,
                                                   const float3 (&gout)[2], float4* gatlas, float* w, float3 (&value)[2]) {
    value[0] = value[1] = f3(0, 0, 0);
    ProbeCell cell;
    if (!probe_cell(position, g, states, &cell)) return;
    const LookupScales s = lookup_scales(g);
    float3 biased[2], S[2], Sf[2];
    float2 nuv[2];
    float W[2], Wf[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        biased[q] = biased_position(position, normal[q], toCamera, g);
        nuv[q] = oct_uv(normal[q]);
        S[q] = Sf[q] = f3(0, 0, 0);
        W[q] = Wf[q] = 0.0f;
    }
    // one lookup's colour at a probe, in square-root space, and its texels
    auto colour = [&](const CellProbe& p, int q, Tap* t) {
        *t = atlas_tap(p.tile + s.cinv, p.z + s.cinv, nuv[q], s.cscale, s.cr, g.color_w, g.color_h);
        float c00[3], c10[3], c01[3], c11[3], r[3];
        at.color.fetch(t->row0, c00);
        at.color.fetch(t->row0 + 1u, c10);
        at.color.fetch(t->row1, c01);
        at.color.fetch(t->row1 + 1u, c11);
        const float w11 = t->ax * t->ay, w10 = t->ax - w11, w01 = t->ay - w11, w00 = 1.0f - t->ax - w01;
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = sqrtf(w00 * c00[k] + w10 * c10[k] + w01 * c01[k] + w11 * c11[k]);
        return f3(r[0], r[1], r[2]);
    };
#pragma unroll 1
    for (uint32_t live = cell.live; live != 0u; live &= live - 1u) {
        const uint32_t i = (uint32_t)__ffs((int)live) - 1u;
        const CellProbe p = cell_probe(cell, i, position, g);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            Tap t;
            const float3 c = colour(p, q, &t);
            float weight, fallback;
            probe_weights(p, p.at - biased[q], normal[q], at.depth, s, g, &weight, &fallback);
            w[(4 * i + 2 * q) * kAdjointThreads] = weight;
            w[(4 * i + 2 * q + 1) * kAdjointThreads] = fallback;
            S[q] = S[q] + c * weight;
            W[q] += weight;
            Sf[q] = Sf[q] + c * fallback;
            Wf[q] += fallback;
        }
    }
    float3 coef[2], coef_f[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float n = W[q] > 1e-3f ? 1.0f / W[q] : 1.0f, nf = Wf[q] > 1e-3f ? 1.0f / Wf[q] : 1.0f;
        const float a = 8.0f * clampf(W[q], 0.0f, 1.0f / 8.0f);
        const float3 fin = S[q] * n, fb = Sf[q] * nf;
        value[q] = mix3(fb * fb, fin * fin, a);
        // d out / d s_i = (1-a) 2 Sf nf^2 wf_i + a 2 S n^2 w_i, per channel
        coef_f[q] = fb * (2.0f * (1.0f - a) * nf) * gout[q];
        coef[q] = fin * (2.0f * a * n) * gout[q];
    }
#pragma unroll 1
    for (uint32_t live = cell.live; live != 0u; live &= live - 1u) {
        const uint32_t i = (uint32_t)__ffs((int)live) - 1u;
        const CellProbe p = cell_probe(cell, i, position, g);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            Tap t;
            const float3 c = colour(p, q, &t);
            const float weight = w[(4 * i + 2 * q) * kAdjointThreads], fallback = w[(4 * i + 2 * q + 1) * kAdjointThreads];
            const float3 ds = coef_f[q] * fallback + coef[q] * weight;  // dL/ds_i
            const float3 dc = f3(c.x > 0.0f ? ds.x / (2.0f * c.x) : 0.0f, c.y > 0.0f ? ds.y / (2.0f * c.y) : 0.0f,
                                 c.z > 0.0f ? ds.z / (2.0f * c.z) : 0.0f);
            const float w11 = t.ax * t.ay, w10 = t.ax - w11, w01 = t.ay - w11, w00 = 1.0f - t.ax - w01;
            float4* p0 = gatlas + t.row0;
            float4* p1 = gatlas + t.row1;
            add_texel(p0, dc.x * w00, dc.y * w00, dc.z * w00);
            if (w10 != 0.0f) add_texel(p0 + 1, dc.x * w10, dc.y * w10, dc.z * w10);
            if (w01 != 0.0f) add_texel(p1, dc.x * w01, dc.y * w01, dc.z * w01);
            if (w11 != 0.0f) add_texel(p1 + 1, dc.x * w11, dc.y * w11, dc.z * w11);
        }
    }
}

// Vector-Jacobian product of pbrMetallicRoughness with respect to albedo
// (pbrMetallicRoughness.glsl:43-84), for a general metalness.
__device__ float3 pbr_albedo_vjp(float3 n, float3 v, float3 lightColor, float3 lightDir, float3 albedo, float metal,
                                 float rough, float3 gout) {
    const float pi = DDGI_PI;
    float3 spec = mix3(f3(0.04f, 0.04f, 0.04f), albedo, metal);
    int jmax = spec.x >= spec.y ? 0 : 1;
    float smax = fmaxf(spec.x, spec.y);
    if (!(smax >= spec.z)) jmax = 2;
    smax = fmaxf(smax, spec.z);
    float r90raw = smax * 25.0f;
    float dr90 = (r90raw > 0.0f && r90raw < 1.0f) ? 25.0f * metal : 0.0f;
    float r90 = clampf(r90raw, 0.0f, 1.0f);
    float alphaRoughness = rough * rough;
    float3 l = norm3(lightDir);
    float3 h = norm3(l + v);
    float NdotL = clampf(dot3(n, l), 0.001f, 1.0f);
    float NdotV = clampf(fabsf(dot3(n, v)), 0.001f, 1.0f);
    float NdotH = clampf(dot3(n, h), 0.0f, 1.0f);
    float VdotH = clampf(dot3(v, h), 0.0f, 1.0f);
    float x = clampf(1.0f - VdotH, 0.0f, 1.0f);
    float x2 = x * x;
    float p5 = x2 * x2 * x;
    float3 F = spec + (f3(r90, r90, r90) - spec) * p5;
    float a2 = alphaRoughness * alphaRoughness;
    float attL = 2.0f * NdotL / (NdotL + sqrtf(a2 + (1.0f - a2) * (NdotL * NdotL)));
    float attV = 2.0f * NdotV / (NdotV + sqrtf(a2 + (1.0f - a2) * (NdotV * NdotV)));
    float a = NdotH * alphaRoughness;
    float k = alphaRoughness / ((1.0f - NdotH * NdotH) + a * a);
    float D = clampf(k * k * (1.0f / pi), 0.0f, 4.0f);
    float GD4 = attL * attV * D / (4.0f * NdotL * NdotV);
    float3 dcol = albedo * (1.0f - 0.04f) * (1.0f - metal);
    float3 e = gout * lightColor * NdotL;
    float3 q = f3(GD4 - dcol.x / pi, GD4 - dcol.y / pi, GD4 - dcol.z / pi);
    float3 ga = f3(e.x * (1.0f - F.x), e.y * (1.0f - F.y), e.z * (1.0f - F.z)) * ((1.0f - 0.04f) * (1.0f - metal) / pi);
    ga = ga + e * q * (metal * (1.0f - p5));
    float sumq = e.x * q.x + e.y * q.y + e.z * q.z;
    float extra = p5 * dr90 * sumq;
    if (jmax == 0) ga.x += extra;
    else if (jmax == 1) ga.y += extra;
    else ga.z += extra;
    return ga;
}

// Parameter gradients and the bounce scatter of every ray of one update.
// grad layout (doubles): albedo [material_count][3], sun [3], sky [3].
__global__ void __launch_bounds__(kAdjointThreads) k_ray_adjoint(DeviceScene sc, DeviceGrid g, DeviceLight L,
                                                     const float4* __restrict__ dirs,
                                                     const uint32_t* __restrict__ states, AtlasF32 at,
                                                     const float4* __restrict__ thit, const uint32_t* __restrict__ prim,
                                                     const float4* __restrict__ gx, float4* gatlas, double* grad,
                                                     uint32_t total, bool smem_albedo, uint32_t* err) {
    extern __shared__ double s_grad[];  // [M*3 if smem_albedo] + sun[3] + sky[3]
    __shared__ float s_weights[kLookupWords][kAdjointThreads];
    const uint32_t M3 = smem_albedo ? sc.material_count * 3 : 0;
    for (uint32_t k = threadIdx.x; k < M3 + 6; k += blockDim.x) s_grad[k] = 0.0;
    __syncthreads();
    double* s_sun = s_grad + M3;
    double* s_sky = s_sun + 3;
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < total) {
        const uint32_t R = g.rays, slot = i / R, ray = i - slot * R;
        float4 th = thit[i];
        uint32_t pb = prim[i], inst = __float_as_uint(th.w);
        float4 gv = gx[i];
        float3 gxi = f3(gv.x, gv.y, gv.z);
        if (inst == 0xFFFFFFFFu) {
            atomicAdd(&s_sky[0], (double)gxi.x);
            atomicAdd(&s_sky[1], (double)gxi.y);
            atomicAdd(&s_sky[2], (double)gxi.z);
        } else if (!(pb & kBackBit) && (gxi.x != 0.0f || gxi.y != 0.0f || gxi.z != 0.0f)) {
            float4 d4 = dirs[ray];
            float3 dir = f3(d4.x, d4.y, d4.z);
            Surface s;
            if (surface_at(sc, probe_origin_exact(g, slot), dir, th.x, th.y, th.z, inst, pb & kPrimMask, &s, err)) {
                const bool shadowed = (pb & kShadowBit) != 0;
                const float fade = night_fade(L);
                const float3 sun = f3(L.color[0], L.color[1], L.color[2]);
                const float3 ldir = f3(L.dir[0], L.dir[1], L.dir[2]);
                float3 spec = mix3(f3(0.04f, 0.04f, 0.04f), s.albedo, s.metal);
                float3 diffuse = s.albedo * (1.0f - 0.04f) * (1.0f - s.metal);
                float3 g_base = shadowed ? gxi : gxi * fade;
                float3 g_pbr = shadowed ? f3(0, 0, 0) : gxi * fade;
                const float3 lookups[2] = {reflected(dir, s.normal), s.normal}, gout[2] = {g_base * spec, g_base * diffuse};
                float3 value[2];  // reflection, indirect
                sample_probes_vjp2(s.position, lookups, -dir, g, states, at, gout, gatlas, &s_weights[0][threadIdx.x],
                                   value);
                const float3 refl = value[0], ind = value[1];
                float3 ga = g_base * (refl * s.metal + ind * ((1.0f - 0.04f) * (1.0f - s.metal)));
                if (!shadowed) {
                    float3 v = norm3(-dir);
                    ga = ga + pbr_albedo_vjp(s.normal, v, sun, ldir, s.albedo, s.metal, s.rough, g_pbr);
                    float3 factor = pbr_metallic_roughness(s.normal, v, f3(1, 1, 1), ldir, s.albedo, s.metal, s.rough);
                    atomicAdd(&s_sun[0], (double)(g_pbr.x * factor.x));
                    atomicAdd(&s_sun[1], (double)(g_pbr.y * factor.y));
                    atomicAdd(&s_sun[2], (double)(g_pbr.z * factor.z));
                }
                double* ag = smem_albedo ? s_grad + 3 * s.material : grad + 3 * (size_t)s.material;
                atomicAdd(ag + 0, (double)ga.x);
                atomicAdd(ag + 1, (double)ga.y);
                atomicAdd(ag + 2, (double)ga.z);
            }
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < M3 + 6; k += blockDim.x) {
        double v = s_grad[k];
        if (v != 0.0) atomicAdd(grad + (k < M3 ? k : sc.material_count * 3 + (k - M3)), v);
    }
}

}  // namespace

cudaError_t launch_replay_update(const DeviceScene& sc, const DeviceGrid& g, const DeviceLight& L, const float4* dirs,
                                 uint32_t* states, float4* color, float2* depth, const float4* thit,
                                 const uint32_t* prim, float4* rays, float* W, float* wsum, uint32_t* err,
                                 cudaStream_t st) {
    const uint32_t P = (uint32_t)(g.res[0] * g.res[1] * g.res[2]);
    const uint32_t total = P * g.rays;
    AtlasF32 at{{color}, {depth}};
    k_replay_shade<<<(total + 127) / 128, 128, 0, st>>>(sc, g, L, dirs, states, at, thit, prim, rays, total, err);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // the kernel with the weights computed once: the same bits as the forward's
    // blend in either pipeline, 0.37 -> 0.06 ms for 2,048 probes of 256 rays
    return launch_blend_fp32_shared(g, nullptr, P, rays, dirs, W, wsum, states, color, depth, st);
}

cudaError_t launch_adjoint_step(const DeviceScene& sc, const DeviceGrid& g, const DeviceLight& L, const float4* dirs,
                                const uint32_t* states, const float4* color_prev, const float2* depth_prev,
                                const float4* thit, const uint32_t* prim, const float4* gk, float4* gprev, float4* gx,
                                float* W, float* wsum, double* grad, uint32_t* err, cudaStream_t st) {
    const uint32_t P = (uint32_t)(g.res[0] * g.res[1] * g.res[2]);
    const uint32_t total = P * g.rays;
    const uint32_t nt = (g.color_res - 2) * (g.color_res - 2);
    cudaError_t e = launch_color_weights(g, dirs, W, wsum, st);
    if (e != cudaSuccess) return e;
    k_blend_adjoint<<<P, 256, sizeof(float) * 6 * nt, st>>>(g, dirs, wsum, gk, gprev, gx);
    AtlasF32 at{{color_prev}, {depth_prev}};
    const bool smem_albedo = sc.material_count <= 1024;
    size_t smem = sizeof(double) * ((smem_albedo ? sc.material_count * 3 : 0) + 6);
    k_ray_adjoint<<<(total + kAdjointThreads - 1) / kAdjointThreads, kAdjointThreads, smem, st>>>(sc, g, L, dirs, states, at, thit, prim, gx, gprev, grad,
                                                          total, smem_albedo, err);
    return cudaGetLastError();
}

}  // namespace ddgi
