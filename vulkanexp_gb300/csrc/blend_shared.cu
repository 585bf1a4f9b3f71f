// blend_shared.cu — FP32 atlas blend with the blend weights computed once per
// update instead of once per probe.
//
// Every probe of an update traces the same direction table, so the weight of
// ray r in interior texel t (max(0, n_t . d_r) for colour, its depth-sharpness
// power for depth: src/shaders/probesUpdate.glsl:71-98) and each texel's
// weight sum are the same for all probes.  k_fp32_weights computes them once
// (W[r][t], texel-contiguous, and the sums in ray order); the blend then is a
// product of each probe's ray records with W, done for two to eight probes per
// block so that each W row is read once per block.  Arithmetic and
// accumulation order per (probe, texel) are those of blend.cu's per-probe
// kernel (common.cuh's blend_* operations, sums in ray order, the same
// normalisation, border copy and probe-state rule), which remains the plain
// reference-like form.
//
// Bound by latency where few probes are blended and by the weights' way from
// L2 where many are.  Measured on GB300 (8/16 tiles) against one thread per
// texel with eight probes a block, scalar sums and weights loaded where they
// are used: 512 probes of 128 rays 149 -> 25 us (weights and blend), 2,048 of
// 256 rays 285 -> 60 us, 16,384 of 256 rays 0.71 -> 0.26 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/ddgi.h"
#include "common.cuh"
#include "kernels.h"

namespace ddgi {

namespace {

// Weights: kWeightTexels texels x 32 rays per 256-thread block.
constexpr uint32_t kWeightTexels = 8;
// Blend: one thread per interior texel, depth and colour texels in warps of
// their own (196 + 36 texels of 16/8 tiles: seven and two warps).
constexpr uint32_t kBlendThreads = 288;
constexpr uint32_t kBatchTile = 4;  // probes per work item of a batch

// Weights of kWeightTexels texels from `t0` over all rays, by one block: a
// thread computes every 32nd ray's weight of one texel (the powers of the
// depth weights are the cost), then eight threads add up the texels' sums in
// ray order from shared memory.  One thread per texel doing both took 31 us
// at 128 rays and 65 us at 256, on two blocks of the whole GPU; 5 and 8 us now.
__device__ __forceinline__ void texel_weights(const DeviceGrid& g, const float4* __restrict__ dirs, uint32_t t0,
                                              float* __restrict__ W, float* __restrict__ wsum) {
    extern __shared__ float s_w[];  // [kWeightTexels][R + 1]
    const int nc = (int)g.color_res - 2, nd = (int)g.depth_res - 2;
    const uint32_t ncol = (uint32_t)(nc * nc), ntex = ncol + (uint32_t)(nd * nd);
    const uint32_t R = g.rays, k = threadIdx.x % kWeightTexels, t = t0 + k;
    if (t < ntex) {
        const bool col = t < ncol;
        const int u = (int)(col ? t : t - ncol), n = col ? nc : nd;
        const int tx = u % n, ty = u / n;
        const float sc = texel_scale((uint32_t)n), ce = 0.5f * (float)(n - 1);
        const float3 td = oct_decode(sc * ((float)tx - ce), sc * ((float)ty - ce));
        for (uint32_t r = threadIdx.x / kWeightTexels; r < R; r += 32) {
            const float4 d = __ldg(dirs + r);
            float w = blend_cosine(td, d);
            if (!col) w = powf(w, g.sharp);
            W[(size_t)r * ntex + t] = w;
            s_w[k * (R + 1) + r] = w;
        }
    }
    __syncthreads();
    if (threadIdx.x < kWeightTexels && t < ntex) {
        const float* w = s_w + k * (R + 1);
        float aw = 0.0f;
#pragma unroll 8
        for (uint32_t r = 0; r < R; ++r) aw += w[r];
        wsum[t] = aw;
    }
}

__global__ void __launch_bounds__(256) k_fp32_weights(DeviceGrid g, const float4* __restrict__ dirs, float* W,
                                                      float* wsum) {
    let_next_launch();
    texel_weights(g, dirs, blockIdx.x * kWeightTexels, W, wsum);
    after_previous();
}

// Words of a ray's records of TP probes in shared memory: r, g, b, depth of
// the TP probes each, and four words that spread consecutive rays over banks.
template <uint32_t TP>
__host__ __device__ constexpr uint32_t record_words() {
    return 4u * TP + 4u;
}

// Weighted sums of one texel over the rays, for NV values of each of TP
// probes.  The probes of a value sit side by side in shared memory, so one
// load brings two or four of them and one packed instruction advances two;
// the next eight rays' weights are on their way while eight are used.
// `step(w, row)` adds ray w's share.
template <class Step>
__device__ __forceinline__ void over_rays(const float* W, uint32_t ntex, uint32_t R, const float* rec,
                                          uint32_t words, Step step) {
    constexpr uint32_t U = 8;
    float w[U], next[U];
    const uint32_t full = R / U * U;
#pragma unroll
    for (uint32_t k = 0; k < U; ++k) next[k] = full ? W[(size_t)k * ntex] : 0.0f;
    for (uint32_t r = 0; r < full; r += U) {
#pragma unroll
        for (uint32_t k = 0; k < U; ++k) w[k] = next[k];
        if (r + U < full) {
#pragma unroll
            for (uint32_t k = 0; k < U; ++k) next[k] = W[(size_t)(r + U + k) * ntex];
        }
#pragma unroll
        for (uint32_t k = 0; k < U; ++k) step(pack2(w[k], w[k]), rec + (size_t)(r + k) * words);
    }
    for (uint32_t r = full; r < R; ++r) {
        const float x = W[(size_t)r * ntex];
        step(pack2(x, x), rec + (size_t)r * words);
    }
}

// TP consecutive probes' values as TP / 2 pairs.
template <uint32_t TP>
__device__ __forceinline__ void load_pairs(const float* p, uint64_t (&v)[TP / 2]) {
    if (TP == 2) {
        v[0] = *reinterpret_cast<const uint64_t*>(p);
    } else {
#pragma unroll
        for (uint32_t j = 0; j < TP / 4; ++j) {
            const ulonglong2 q = reinterpret_cast<const ulonglong2*>(p)[j];
            v[2 * j] = q.x;
            v[2 * j + 1] = q.y;
        }
    }
}

// Blend of probes p0 .. p0 + np - 1 (slots of `rays`) by one block.  The records
// and the weights come from kernels that can still be running when this one is
// set up, so their pointers are not declared to be read-only throughout.
template <uint32_t TP>
__device__ __forceinline__ void blend_probes_shared(const DeviceGrid& g, const uint32_t* probe_list, uint32_t p0,
                                                    uint32_t np, const float4* rays, const float* W,
                                                    const float* wsum, uint32_t* states, float4* color,
                                                    float2* depth, const float hy) {
    extern __shared__ float4 s_dyn[];
    float* const s_rec = reinterpret_cast<float*>(s_dyn);  // [R][record_words]: colour, clamped depth
    __shared__ uint32_t s_max_change[TP], s_out_of_range[TP], s_probe[TP];
    constexpr uint32_t words = record_words<TP>();
    const uint32_t R = g.rays;
    const float cl = g.cell_len;
    if (threadIdx.x < TP) {
        s_max_change[threadIdx.x] = 0u;
        s_out_of_range[threadIdx.x] = 0u;
        s_probe[threadIdx.x] = threadIdx.x < np ? (probe_list ? probe_list[p0 + threadIdx.x] : p0 + threadIdx.x) : 0u;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < TP * R; i += blockDim.x) {
        const uint32_t p = i / R, r = i - p * R;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (p < np) {
            v = rays[(size_t)p0 * R + i];
            if (v.w < 0.0f || v.w > cl) atomicAdd(&s_out_of_range[p], 1u);
            v.w = fminf(cl, v.w);
            if (v.w < 0.0f) v.w = cl;
        }
        float* q = s_rec + (size_t)r * words + p;
        q[0] = v.x;
        q[TP] = v.y;
        q[2 * TP] = v.z;
        q[3 * TP] = v.w;
    }
    __syncthreads();

    const uint32_t rx = (uint32_t)g.res[0], rxy = (uint32_t)(g.res[0] * g.res[1]);
    const int nc = (int)g.color_res - 2, nd = (int)g.depth_res - 2;
    const uint32_t ncol = (uint32_t)(nc * nc), ndep = (uint32_t)(nd * nd), ntex = ncol + ndep;
    const uint32_t dep_items = (ndep + 31u) & ~31u, items = dep_items + ((ncol + 31u) & ~31u);
    for (uint32_t item = threadIdx.x; item < items; item += blockDim.x) {
        if (item < dep_items) {
            if (item >= ndep) continue;
            uint64_t a0[TP / 2], a1[TP / 2];
#pragma unroll
            for (uint32_t j = 0; j < TP / 2; ++j) a0[j] = a1[j] = 0u;
            over_rays(W + ncol + item, ntex, R, s_rec + 3 * TP, words, [&](uint64_t w, const float* row) {
                uint64_t dep[TP / 2];
                load_pairs<TP>(row, dep);
#pragma unroll
                for (uint32_t j = 0; j < TP / 2; ++j) {  // blend_add, blend_add_square
                    a0[j] = fma2(w, dep[j], a0[j]);
                    a1[j] = fma2(mul2(w, dep[j]), dep[j], a1[j]);
                }
            });
            const float aw = wsum[ncol + item];
            const int tx = (int)item % nd, ty = (int)item / nd;
#pragma unroll
            for (uint32_t p = 0; p < TP; ++p) {
                if (p >= np) continue;
                float lo, hi, m0, m1;
                unpack2(a0[p / 2], &lo, &hi);
                m0 = p & 1 ? hi : lo;
                unpack2(a1[p / 2], &lo, &hi);
                m1 = p & 1 ? hi : lo;
                if (aw > 1e-3f) {
                    m0 /= aw;
                    m1 /= aw;
                }
                const uint32_t probe = s_probe[p];
                const int ix = (int)(probe % rx), iy = (int)((probe % rxy) / rx), iz = (int)(probe / rxy);
                const int tile = iy * g.res[0] + ix;
                size_t px = (size_t)((int)g.depth_res * tile + 1 + tx), py = (size_t)((int)g.depth_res * iz + 1 + ty);
                float2* texel = depth + py * g.depth_w + px;
                float2 prev = *texel;
                *texel = store_depth(g, blend_hysteresis(m0, prev.x, hy), blend_hysteresis(m1, prev.y, hy));
            }
        } else {
            const uint32_t t = item - dep_items;
            if (t >= ncol) continue;
            uint64_t a[3][TP / 2];
#pragma unroll
            for (uint32_t j = 0; j < TP / 2; ++j) a[0][j] = a[1][j] = a[2][j] = 0u;
            over_rays(W + t, ntex, R, s_rec, words, [&](uint64_t w, const float* row) {
#pragma unroll
                for (uint32_t c = 0; c < 3; ++c) {
                    uint64_t v[TP / 2];
                    load_pairs<TP>(row + c * TP, v);
#pragma unroll  // blend_add
                    for (uint32_t j = 0; j < TP / 2; ++j) a[c][j] = fma2(w, v[j], a[c][j]);
                }
            });
            const float aw = wsum[t];
            const int tx = (int)t % nc, ty = (int)t / nc;
#pragma unroll
            for (uint32_t p = 0; p < TP; ++p) {
                if (p >= np) continue;
                float m[3];
#pragma unroll
                for (uint32_t c = 0; c < 3; ++c) {
                    float lo, hi;
                    unpack2(a[c][p / 2], &lo, &hi);
                    m[c] = p & 1 ? hi : lo;
                    if (aw > 1e-3f) m[c] /= aw;
                }
                const uint32_t probe = s_probe[p];
                const int ix = (int)(probe % rx), iy = (int)((probe % rxy) / rx), iz = (int)(probe / rxy);
                const int tile = iy * g.res[0] + ix;
                size_t px = (size_t)((int)g.color_res * tile + 1 + tx), py = (size_t)((int)g.color_res * iz + 1 + ty);
                float4* texel = color + py * g.color_w + px;
                float4 prev = *texel;
                float mc = fmaxf(fmaxf(fabsf(m[0] - prev.x), fabsf(m[1] - prev.y)), fabsf(m[2] - prev.z));
                atomicMax(&s_max_change[p], __float_as_uint(mc));
                *texel = store_color(g, blend_hysteresis(m[0], prev.x, hy), blend_hysteresis(m[1], prev.y, hy),
                                     blend_hysteresis(m[2], prev.z, hy));
            }
        }
    }
    __syncthreads();

    // border copy (probesCopyBorders.comp, generalised) of each probe
    const int nbc = 4 + 4 * nc, nbd = 4 + 4 * nd;
    for (uint32_t i = threadIdx.x; i < np * (uint32_t)(nbc + nbd); i += blockDim.x) {
        const uint32_t p = i / (uint32_t)(nbc + nbd);
        const int e = (int)(i % (uint32_t)(nbc + nbd));
        const uint32_t probe = s_probe[p];
        const int ix = (int)(probe % rx), iy = (int)((probe % rxy) / rx), iz = (int)(probe / rxy);
        const int tile = iy * g.res[0] + ix;
        if (e < nbc) {
            int4 b = border_entry(e, (int)g.color_res);
            size_t ox = (size_t)g.color_res * tile, oy = (size_t)g.color_res * iz;
            color[(oy + b.y) * g.color_w + ox + b.x] = color[(oy + b.w) * g.color_w + ox + b.z];
        } else {
            int4 b = border_entry(e - nbc, (int)g.depth_res);
            size_t ox = (size_t)g.depth_res * tile, oy = (size_t)g.depth_res * iz;
            depth[(oy + b.y) * g.depth_w + ox + b.x] = depth[(oy + b.w) * g.depth_w + ox + b.z];
        }
    }

    if (threadIdx.x < np) {  // probesUpdate.glsl:110-119
        const uint32_t p = threadIdx.x, probe = s_probe[p];
        uint32_t s = states[probe];
        if (s_out_of_range[p] >= R) {
            s = 8;
        } else {
            float mc = __uint_as_float(s_max_change[p]);
            float sf = (float)s;
            if (mc < 0.02f / sf) s = min(s + 1u, 8u);
            else if (mc > 0.04f / sf) s = max(s - 1u, 1u);
            else if (mc > 0.25f) s = 1;
        }
        states[probe] = s;
    }
}

// Probes per block for n listed probes, chosen on the device (a scheduled
// update's count is known only there): the most of 8, 4, 2 that still gives
// every SM's three resident blocks a tile.  A block's time hardly depends on
// its probes (a serial sum over the rays), so few probes want many blocks;
// many probes want each weight row read for as many of them as possible.
__device__ __forceinline__ uint32_t probes_per_block(uint32_t n, uint32_t slots) {
    return n >= 8u * slots ? 8u : (n >= 4u * slots ? 4u : 2u);
}

__global__ void __launch_bounds__(kBlendThreads, 3) k_blend_fp32_shared(DeviceGrid g, const uint32_t* probe_list,
                                                                        uint32_t nprobes, const float4* rays,
                                                                        const float* W, const float* wsum,
                                                                        uint32_t* states, float4* color, float2* depth,
                                                                        const uint32_t* dev_count,
                                                                        const float* hyst_dev, uint32_t slots) {
    after_previous();
    const uint32_t n = dev_count ? min(*dev_count, nprobes) : nprobes;
    const uint32_t tp = probes_per_block(n, slots);
    const float hy = hyst_dev ? *hyst_dev : g.hyst;
    for (uint32_t p0 = blockIdx.x * tp; p0 < n; p0 += gridDim.x * tp) {
        const uint32_t np = min(tp, n - p0);
        if (tp == 8u)
            blend_probes_shared<8>(g, probe_list, p0, np, rays, W, wsum, states, color, depth, hy);
        else if (tp == 4u)
            blend_probes_shared<4>(g, probe_list, p0, np, rays, W, wsum, states, color, depth, hy);
        else
            blend_probes_shared<2>(g, probe_list, p0, np, rays, W, wsum, states, color, depth, hy);
        __syncthreads();  // the next tile reuses the shared memory
    }
}

// Batched form: weights per FP32 volume (grid y = position in the list),
// then block b blends tile (b - tile_base[i]) of kBatchTile probes of
// volume list[i]; the block finishing a volume's last tile stamps its
// completion time.
__global__ void __launch_bounds__(256) k_batch_fp32_weights(BatchTables bt, BatchBlendList bl) {
    const BatchVolume& vol = bt.vols[__ldg(bl.list + blockIdx.y)];
    texel_weights(vol.g, bt.dirs + vol.dir_base, blockIdx.x * kWeightTexels,
                  reinterpret_cast<float*>(vol.wbuf), vol.rowsum);
}

__global__ void __launch_bounds__(kBlendThreads, 3) k_batch_blend_fp32_shared(BatchTables bt, BatchBlendList bl,
                                                                              const float4* __restrict__ rays) {
    uint32_t lo = 0, hi = bl.n;  // tile_base[lo] <= b < tile_base[hi]
    const uint32_t b = blockIdx.x;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(bl.tile_base + mid) <= b) lo = mid;
        else hi = mid;
    }
    const uint32_t v = __ldg(bl.list + lo);
    const BatchVolume& vol = bt.vols[v];
    const uint32_t P = (uint32_t)vol.g.res[0] * (uint32_t)vol.g.res[1] * (uint32_t)vol.g.res[2];
    const uint32_t p0 = (b - __ldg(bl.tile_base + lo)) * kBatchTile;
    if (p0 < P)
        blend_probes_shared<kBatchTile>(vol.g, nullptr, p0, min(kBatchTile, P - p0), rays + vol.ray_base,
                                        reinterpret_cast<const float*>(vol.wbuf), vol.rowsum, vol.states,
                                        static_cast<float4*>(vol.color), static_cast<float2*>(vol.depth), vol.g.hyst);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t items = __ldg(bl.tile_base + lo + 1) - __ldg(bl.tile_base + lo);
        if (atomicAdd(bt.done + v, 1u) == items - 1u) bt.clock[1 + v] = globaltimer_ns();
    }
}

}  // namespace

size_t fp32_weight_bytes(uint32_t rays, uint32_t color_res, uint32_t depth_res) {
    const size_t ntex = (size_t)(color_res - 2) * (color_res - 2) + (size_t)(depth_res - 2) * (depth_res - 2);
    return ntex * rays * sizeof(float);
}

uint32_t fp32_shared_tiles(uint32_t nprobes) { return (nprobes + kBatchTile - 1) / kBatchTile; }

namespace {

size_t weight_smem(uint32_t rays) { return sizeof(float) * kWeightTexels * (rays + 1); }
template <uint32_t TP>
size_t blend_smem(uint32_t rays) {
    return sizeof(float) * record_words<TP>() * rays;
}
uint32_t weight_blocks(uint32_t ntex) { return (ntex + kWeightTexels - 1) / kWeightTexels; }

}  // namespace

// Record staging and weight rows at up to DDGI_MAX_RAYS_PER_PROBE rays, on
// the current device.
cudaError_t set_shared_smem_limit() {
    cudaError_t e = ensure_dynamic_smem(k_blend_fp32_shared, (int)blend_smem<8>(DDGI_MAX_RAYS_PER_PROBE));
    if (e == cudaSuccess)
        e = ensure_dynamic_smem(k_batch_blend_fp32_shared, (int)blend_smem<kBatchTile>(DDGI_MAX_RAYS_PER_PROBE));
    return e;
}

cudaError_t launch_color_weights(const DeviceGrid& g, const float4* dirs, float* W, float* wsum, cudaStream_t st) {
    // the colour texels come first; a last block's depth texels do no harm
    k_fp32_weights<<<weight_blocks((g.color_res - 2) * (g.color_res - 2)), 256, weight_smem(g.rays), st>>>(g, dirs, W,
                                                                                                         wsum);
    return cudaGetLastError();
}

cudaError_t launch_blend_fp32_shared(const DeviceGrid& g, const uint32_t* probe_list, uint32_t nprobes,
                                     const float4* rays, const float4* dirs, float* W, float* wsum, uint32_t* states,
                                     float4* color, float2* depth, cudaStream_t st, const uint32_t* dev_count,
                                     const float* hyst_dev, bool early_weights) {
    if (nprobes == 0) return cudaSuccess;
    cudaError_t e = set_shared_smem_limit();
    if (e != cudaSuccess) return e;
    const uint32_t ntex = (g.color_res - 2) * (g.color_res - 2) + (g.depth_res - 2) * (g.depth_res - 2);
    if (early_weights)
        e = launch_dependent(k_fp32_weights, weight_blocks(ntex), 256, weight_smem(g.rays), st, g, dirs, W, wsum);
    else
        k_fp32_weights<<<weight_blocks(ntex), 256, weight_smem(g.rays), st>>>(g, dirs, W, wsum);
    if (e != cudaSuccess) return e;
    const uint32_t slots = 3u * sm_count();
    // the most probes a block can be given decides its shared memory
    const size_t smem = nprobes >= 8u * slots ? blend_smem<8>(g.rays)
                                              : (nprobes >= 4u * slots ? blend_smem<4>(g.rays) : blend_smem<2>(g.rays));
    e = launch_dependent(k_blend_fp32_shared, min((nprobes + 1u) / 2u, slots), kBlendThreads, smem, st, g, probe_list,
                         nprobes, rays, W, wsum, states, color, depth, dev_count, hyst_dev, slots);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_batch_blend_fp32_shared(const BatchTables& bt, const BatchBlendList& bl, uint32_t max_ntex,
                                           uint32_t max_rays, const float4* rays, cudaStream_t st) {
    if (bl.ntiles == 0) return cudaSuccess;
    cudaError_t e = set_shared_smem_limit();
    if (e != cudaSuccess) return e;
    k_batch_fp32_weights<<<dim3(weight_blocks(max_ntex), bl.n), 256, weight_smem(max_rays), st>>>(bt, bl);
    k_batch_blend_fp32_shared<<<bl.ntiles, kBlendThreads, blend_smem<kBatchTile>(max_rays), st>>>(bt, bl, rays);
    return cudaGetLastError();
}

}  // namespace ddgi
