// wavefront.cu — the probe trace as three kernels instead of one.
//
//  1. k_primary: closest hit of every probe ray.  Persistent warps; a lane
//     whose ray finishes is handed the next ray from a global counter, so the
//     warp keeps its lanes busy instead of waiting for its longest ray.
//  2. k_shade_classify, k_shade_front: one thread per ray record, coalesced:
//     miss -> sky, backface -> (0, 0.8 t), front face -> a queue that is shaded
//     with one to four lanes per hit, up to the shadow query; the front hits
//     are appended (warp-aggregated) to a shadow-ray queue.
//  3. k_shadow: any-hit query of the queued rays toward the sun, persistent
//     like k_primary; an unshadowed ray gets (base + sun) * fade.
//
// Results are identical to the single fused kernel (same traversal, same
// shading arithmetic); only the schedule differs.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "shade.cuh"
#include "traverse.cuh"

namespace ddgi {

namespace {

constexpr int kPersistThreads = kWalkerThreads;  // the walkers' shared-memory stacks assume it
constexpr uint32_t kShadeBlocksPerSm = 5;  // resident blocks of the front-hit shading
constexpr unsigned kFull = 0xffffffffu;

// Work item `id` of a grouped order: groups of G = 32 / rpw probes (in perm
// order) take rpw consecutive directions of the ray order each per 32 items,
// so a warp traces similar directions from neighbouring probes.  Returns the
// probe slot and the position in the ray order.
__device__ __forceinline__ void grouped_ray(uint32_t id, uint32_t R, uint32_t rpw, uint32_t n,
                                            const uint32_t* perm, uint32_t* slot, uint32_t* j) {
    const uint32_t G = 32u / rpw;
    const uint32_t first = (id / (G * R)) * G;
    const uint32_t m = min(G, n - first);
    const uint32_t local = id - first * R;
    const uint32_t span = m * rpw;
    const uint32_t c = local / span, r = local - c * span;
    const uint32_t q = r / rpw;
    *j = c * rpw + (r - q * rpw);
    *slot = __ldg(perm + first + q);
}

struct PrimaryJob {
    static constexpr float kTmin = 0.01f;
    static constexpr uint32_t kMask = 0x3u;
    DeviceGrid g;
    const uint32_t* probe_list;
    const float4* dirs;
    const uint32_t* ray_order;
    WaveHits hits;
    uint32_t total;
    const uint32_t* dev_count;  // listed probes, read on the device (NULL: total / rays)
    const uint32_t* perm;       // grouped order over all probes (NULL: a warp per probe slot)
    uint32_t rpw, nprobes;

    template <class W>
    __device__ __forceinline__ bool start(W& w, const DeviceScene& sc, uint32_t id, uint32_t* out) const {
        const uint32_t R = g.rays;
        uint32_t slot, j;
        if (perm) {
            grouped_ray(id, R, rpw, nprobes, perm, &slot, &j);
        } else {
            slot = id / R;
            j = id - slot * R;
        }
        uint32_t ray = __ldg(ray_order + j);
        uint32_t probe = probe_list ? __ldg(probe_list + slot) : slot;
        *out = slot * R + ray;
        float4 d4 = __ldg(dirs + ray);
        return w.start(sc, probe_origin_exact(g, probe), f3(d4.x, d4.y, d4.z), g.tmax);
    }
    template <class W>
    __device__ __forceinline__ void finish(const W& w, uint32_t out) const {
        const HitRec& h = w.best;
        hits.thit[out] = make_float4(h.t, h.b1, h.b2, __uint_as_float(h.inst));
        hits.prim[out] = h.prim | (h.back ? 0x80000000u : 0u);
    }
};

struct ShadowJob {
    static constexpr float kTmin = 0.1f;
    static constexpr uint32_t kMask = 0xFFu;
    const ShadowQueue q;
    float3 dir;
    float4* rays;
    uint32_t* prim;  // hit words: bit 30 marks a shadowed front hit (kept for replays)
    uint32_t total;

    template <class W>
    __device__ __forceinline__ bool start(W& w, const DeviceScene& sc, uint32_t id, uint32_t* out) const {
        *out = id;
        float4 p = q.pos[id];
        return w.start(sc, f3(p.x, p.y, p.z), dir, 10000.0f);
    }
    template <class W>
    __device__ __forceinline__ void finish(const W& w, uint32_t id) const {
        uint32_t idx = q.idx[id];
        if (w.best.inst != kNoHit) {  // shadowed: the record keeps the base colour
            prim[idx] |= 1u << 30;
            return;
        }
        float4 sun = q.sun[id];
        float4 rec = rays[idx];
        float3 c = (f3(rec.x, rec.y, rec.z) + f3(sun.x, sun.y, sun.z)) * sun.w;
        rays[idx] = make_float4(c.x, c.y, c.z, rec.w);
    }
};

__device__ __forceinline__ void init_stack(SmemStack& s, int* base, int, int*) { s.base = base; }
__device__ __forceinline__ void init_stack(SplitStack& s, int* base, int split, int* spill) {
    s.base = base;
    s.split = split;
    s.spill = spill;
}
template <class Stack>
struct SpillArea {  // local-memory tail of a SplitStack
    __device__ __forceinline__ int* ptr() { return nullptr; }
};
template <>
struct SpillArea<SplitStack> {
    int a[kSpillMax];
    __device__ __forceinline__ int* ptr() { return a; }
};

// Persistent traversal loop with per-lane refill.  A warp refills when at
// least `refill` of its lanes are idle (or all are), taking as many rays as
// it has idle lanes with one atomic.
template <bool ANY, class Stack, template <bool, class> class Walker, class Job>
__device__ __forceinline__ void persistent_walk(const DeviceScene& sc, const Job& job, uint32_t total,
                                                uint32_t* counter, int stack_cap, int split, WalkKnobs knobs,
                                                uint32_t* err) {
    const int refill = knobs.refill;
    extern __shared__ int s_stack[];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    SpillArea<Stack> spill;
    Walker<ANY, Stack> w;
    init_stack(w.stk, s_stack + threadIdx.x, split, spill.ptr());
    w.cap = stack_cap;
    w.clear();
    w.wait_max = knobs.wait;
    w.tmin = Job::kTmin;
    w.mask = Job::kMask;
    bool active = false;
    bool drained = false;  // warp-uniform: the work counter has passed `total`
    uint32_t out = 0;
    for (uint32_t calls = 0;; ++calls) {
        unsigned busy = __ballot_sync(kFull, active);
        const unsigned idle = ~busy;
        if (!drained && (__popc(idle) >= refill || busy == 0)) {
            int leader = __ffs(idle) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(idle));
            base = __shfl_sync(kFull, base, leader);
            drained = base >= total;  // the counter only grows: every later request fails too
            if (!active) {
                uint32_t id = base + (uint32_t)__popc(idle & lt);
                if (id < total) {
                    if (job.start(w, sc, id, &out)) active = true;
                    else job.finish(w, out);  // empty scene: immediate miss
                }
            }
            busy = __ballot_sync(kFull, active);
        }
        if (busy == 0) {
            if (drained) break;
            continue;
        }
        bool fin = w.advance(sc, err, active, calls);  // every lane takes part (warp votes)
        if (active && fin) {
            job.finish(w, out);
            active = false;
        }
    }
}

template <class Stack, template <bool, class> class Walker>
__global__ void __launch_bounds__(kPersistThreads, Walker<false, Stack>::kMinBlocks) k_primary(DeviceScene sc, PrimaryJob job, uint32_t* counter,
                                                                int stack_cap, int split, WalkKnobs knobs, uint32_t* err) {
    const uint32_t total = job.dev_count ? *job.dev_count * job.g.rays : job.total;
    persistent_walk<false, Stack, Walker>(sc, job, total, counter, stack_cap, split, knobs, err);
}

template <class Stack, template <bool, class> class Walker>
__global__ void __launch_bounds__(kPersistThreads, Walker<false, Stack>::kMinBlocks) k_shadow(DeviceScene sc, ShadowJob job, const uint32_t* qcount,
                                                               uint32_t* counter, int stack_cap, int split, WalkKnobs knobs,
                                                               uint32_t* err) {
    after_previous();
    let_next_launch();  // the blend weights start in the places that the last rays leave
    persistent_walk<true, Stack, Walker>(sc, job, *qcount, counter, stack_cap, split, knobs, err);
}

// Warp-aggregated append: the lanes with `flag` get consecutive slots of a
// queue whose length is *count; returns this lane's slot (valid if flag).
__device__ __forceinline__ uint32_t warp_append(bool flag, uint32_t* count) {
    const unsigned m = __ballot_sync(kFull, flag);
    if (!m) return 0;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(kFull, base, leader);
    return base + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// The same for all threads of a block of kClassifyThreads, which call it
// together, with one atomic per block: of one per warp, 131,072 of them on one
// address were the time of the classification of 4.19 M records (82 -> 31 us).
constexpr uint32_t kClassifyThreads = 512;
__device__ __forceinline__ uint32_t block_append(bool flag, uint32_t* count) {
    constexpr uint32_t kWarps = kClassifyThreads / 32;
    __shared__ uint32_t s_first[kWarps];  // flags per warp, then the warp's first slot
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(kFull, flag);
    if (lane == 0) s_first[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (warp == 0) {
        const uint32_t own = lane < kWarps ? s_first[lane] : 0u;
        uint32_t sum = own;
#pragma unroll
        for (uint32_t o = 1; o < kWarps; o <<= 1) {
            const uint32_t below = __shfl_up_sync(kFull, sum, o);
            if (lane >= o) sum += below;
        }
        uint32_t base = 0;
        if (lane == kWarps - 1 && sum) base = atomicAdd(count, sum);
        base = __shfl_sync(kFull, base, kWarps - 1);
        if (lane < kWarps) s_first[lane] = base + sum - own;
    }
    __syncthreads();
    return s_first[warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// Shading, pass 1, one thread per record: a miss gets the sky radiance
// (miss.rmiss:17-23), a back face (0, 0, 0, 0.8 t) (closesthit.glsl:137-141);
// front faces go to a compacted queue so that pass 2 runs in full warps.
__global__ void __launch_bounds__(kClassifyThreads) k_shade_classify(DeviceGrid g, DeviceLight L, uint32_t total, WaveHits hits,
                                                        float4* rays_out, ddgi_hit* hits_out, uint32_t* front_count,
                                                        const uint32_t* dev_count) {
    after_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (dev_count) total = *dev_count * g.rays;
    bool is_front = false;
    if (i < total) {
        const float4 th = hits.thit[i];
        const uint32_t pb = hits.prim[i];
        const uint32_t inst = __float_as_uint(th.w), prim = pb & 0x0fffffffu;
        const bool back = (pb >> 31) != 0;
        if (inst == kNoHit) rays_out[i] = make_float4(L.sky[0], L.sky[1], L.sky[2], -1.0f);
        else if (back) rays_out[i] = make_float4(0.0f, 0.0f, 0.0f, th.x * 0.80f);
        else is_front = true;
        if (hits_out) {
            ddgi_hit hr;
            hr.instance = inst;
            hr.primitive = inst == kNoHit ? 0u : prim;
            hr.t = inst == kNoHit ? 0.0f : th.x;
            hr.backface = (inst != kNoHit && back) ? 1u : 0u;
            hits_out[i] = hr;
        }
    }
    const uint32_t k = block_append(is_front, front_count);
    if (is_front) hits.front[k] = i;
}

// Shading, pass 2, one thread per queued front hit: closesthit.glsl
// (NO_REFLECTION) up to the shadow query, whose rays are appended to the
// shadow queue (an unshadowed ray later adds the sun term).
// Built for five resident blocks per SM (96 registers): 366 us for the hits of
// the 1M-triangle terrain update against 373 us at six and 396 us at four; 23,
// 25 and 22 us for the 65 K hits of a small room.
template <class AV>
__global__ void __launch_bounds__(128, kShadeBlocksPerSm) k_shade_front(DeviceScene sc, DeviceGrid g, DeviceLight L,
                                                        const uint32_t* __restrict__ probe_list,
                                                        const float4* __restrict__ dirs,
                                                        const uint32_t* __restrict__ states, AV at, WaveHits hits,
                                                        const uint32_t* front_count, float4* rays_out, ShadowQueue q,
                                                        uint32_t* err) {
    after_previous();
    const uint32_t n = *front_count;
    if (blockIdx.x * blockDim.x >= n) return;  // whole block
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    bool enqueue = false;
    SurfaceShade s;
    uint32_t i = 0;
    if (k < n) {
        i = hits.front[k];
        const uint32_t R = g.rays;
        const uint32_t slot = i / R, ray = i - slot * R;
        const float4 th = hits.thit[i];
        const uint32_t inst = __float_as_uint(th.w), prim = hits.prim[i] & 0x0fffffffu;
        const uint32_t probe = probe_list ? __ldg(probe_list + slot) : slot;
        const float4 d4 = __ldg(dirs + ray);
        if (shade_surface(sc, g, L, states, at, probe_origin_exact(g, probe), f3(d4.x, d4.y, d4.z), th.x, th.y, th.z,
                          inst, prim, &s, err))
            enqueue = true;
        rays_out[i] = make_float4(s.base.x, s.base.y, s.base.z, th.x);
    }
    const uint32_t qk = warp_append(enqueue, q.count);
    if (enqueue) {
        q.idx[qk] = i;
        q.pos[qk] = make_float4(s.position.x, s.position.y, s.position.z, 0.0f);
        q.sun[qk] = make_float4(s.sun.x, s.sun.y, s.sun.z, s.fade);
    }
}

// ---------------------------------------------------------------------------
// Probe classification (src/shaders/probesInit.rgen:31-64 with
// probeInitMiss.rmiss and backfaceTest.rchit): 512 closest-hit rays per
// probe among INSTANCE_STATIC (mask 1) instances, t in [0.01, 1.5 |cell|].
// A hit closer than |cell| counts as a back-face hit when back-facing, and
// marks the probe as near geometry when it lies within one cell of the probe
// on every axis (hit position rounded product, then sum).
// ---------------------------------------------------------------------------
struct InitJob {
    static constexpr float kTmin = 0.01f;
    static constexpr uint32_t kMask = 0x1u;
    DeviceGrid g;
    const float4* dirs;  // kInitRays directions
    float tmax;
    uint32_t* back;  // per probe
    uint32_t* near;  // per probe

    template <class W>
    __device__ __forceinline__ bool start(W& w, const DeviceScene& sc, uint32_t id, uint32_t* out) const {
        *out = id;
        const uint32_t probe = id / kInitRays, i = id - probe * kInitRays;
        float4 d4 = __ldg(dirs + i);
        return w.start(sc, probe_origin_exact(g, probe), f3(d4.x, d4.y, d4.z), tmax);
    }
    template <class W>
    __device__ __forceinline__ void finish(const W& w, uint32_t id) const {
        const HitRec& h = w.best;
        if (h.inst == kNoHit || !(h.t < g.cell_len)) return;
        const uint32_t probe = id / kInitRays;
        if (h.back) atomicAdd(back + probe, 1u);
        const float3 o = w.wr.o, d = w.wr.d;
        const float dx = fabsf(__fsub_rn(__fadd_rn(__fmul_rn(d.x, h.t), o.x), o.x));
        const float dy = fabsf(__fsub_rn(__fadd_rn(__fmul_rn(d.y, h.t), o.y), o.y));
        const float dz = fabsf(__fsub_rn(__fadd_rn(__fmul_rn(d.z, h.t), o.z), o.z));
        if (dx < g.cell[0] && dy < g.cell[1] && dz < g.cell[2]) near[probe] = 1u;
    }
};

__global__ void __launch_bounds__(kPersistThreads) k_init_probes(DeviceScene sc, InitJob job, uint32_t total,
                                                                 uint32_t* counter, int stack_cap, uint32_t* err) {
    persistent_walk<false, SmemStack, WarpWalker>(sc, job, total, counter, stack_cap, stack_cap,
                                                  WalkKnobs{8, kDefaultWait}, err);
}

// State per probe: OFF (0) when more than half of raysPerProbe back-face
// hits, else 1 near geometry, else 8.
__global__ void k_init_states(uint32_t P, uint32_t R, const uint32_t* back, const uint32_t* near, uint32_t* states) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    states[p] = 2u * back[p] > R ? 0u : (near[p] ? 1u : 8u);
}

// ---------------------------------------------------------------------------
// Batched form: the records of all volumes form one index space; the volume
// of record `id` is found by binary search of the record offsets.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t batch_volume(const BatchTables& bt, uint32_t id) {
    uint32_t lo = 0, hi = bt.nvol;  // ray_base[lo] <= id < ray_base[hi]
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(bt.ray_base + mid) <= id) lo = mid;
        else hi = mid;
    }
    return lo;
}

struct BatchPrimaryJob {
    static constexpr float kTmin = 0.01f;
    static constexpr uint32_t kMask = 0x3u;
    BatchTables bt;
    WaveHits hits;

    template <class W>
    __device__ __forceinline__ bool start(W& w, const DeviceScene& sc, uint32_t id, uint32_t* out) const {
        id += bt.first;  // records of the launch's volumes
        const uint32_t v = batch_volume(bt, id);
        const BatchVolume& vol = bt.vols[v];
        const uint32_t R = vol.g.rays;
        const uint32_t base = __ldg(bt.ray_base + v);
        const uint32_t local = id - base;
        uint32_t slot, j;
        if (vol.perm) {
            grouped_ray(local, R, vol.rays_per_warp,
                        (uint32_t)vol.g.res[0] * (uint32_t)vol.g.res[1] * (uint32_t)vol.g.res[2], vol.perm, &slot, &j);
        } else {
            slot = local / R;
            j = local - slot * R;
        }
        const uint32_t ray = __ldg(bt.ray_order + vol.dir_base + j);
        *out = base + slot * R + ray;
        float4 d4 = __ldg(bt.dirs + vol.dir_base + ray);
        return w.start_at(sc, W::kWide ? vol.wroot : vol.root, probe_origin_exact(vol.g, slot), f3(d4.x, d4.y, d4.z),
                          vol.g.tmax);
    }
    template <class W>
    __device__ __forceinline__ void finish(const W& w, uint32_t out) const {
        const HitRec& h = w.best;
        hits.thit[out] = make_float4(h.t, h.b1, h.b2, __uint_as_float(h.inst));
        hits.prim[out] = h.prim | (h.back ? 0x80000000u : 0u);
    }
};

// The same with 2 x PARTS lanes per hit: half of them for each of its two
// lookups, in which each takes every PARTS-th probe (the rest of the hit is
// done by all).  With fewer hits than the chip has threads for, the time is one
// thread's chain of eight probes' loads and quotients, which this shortens:
// the 65 K hits of 512 probes 26 -> 17 us, 16 K 20 -> 11 us.
template <int PARTS, class AV>
__global__ void __launch_bounds__(128, kShadeBlocksPerSm) k_shade_front_split(DeviceScene sc, DeviceGrid g, DeviceLight L,
                                                              const uint32_t* __restrict__ probe_list,
                                                              const float4* __restrict__ dirs,
                                                              const uint32_t* __restrict__ states, AV at,
                                                              WaveHits hits, const uint32_t* front_count,
                                                              float4* rays_out, ShadowQueue q, uint32_t* err) {
    constexpr uint32_t kLanes = 2u * PARTS;
    after_previous();
    const uint32_t n = *front_count;
    if (blockIdx.x * (blockDim.x / kLanes) >= n) return;  // whole block
    const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes, lane = threadIdx.x % kLanes;
    bool ok = false;
    Surface s;
    s.position = s.normal = f3(0, 0, 0);
    float3 dir = f3(0, 0, 0);
    uint32_t i = 0;
    float t = 0.0f;
    if (k < n) {
        i = hits.front[k];
        const uint32_t R = g.rays;
        const uint32_t slot = i / R, ray = i - slot * R;
        const float4 th = hits.thit[i];
        const uint32_t inst = __float_as_uint(th.w), prim = hits.prim[i] & 0x0fffffffu;
        const uint32_t probe = probe_list ? __ldg(probe_list + slot) : slot;
        const float4 d4 = __ldg(dirs + ray);
        dir = f3(d4.x, d4.y, d4.z);
        t = th.x;
        ok = surface_at(sc, probe_origin_exact(g, probe), dir, th.x, th.y, th.z, inst, prim, &s, err);
    }
    const float3 mine = sample_probes_split<PARTS>(ok, s.position, lane < PARTS ? reflected(dir, s.normal) : s.normal,
                                                   -dir, g, states, at);
    const float3 other = f3(__shfl_xor_sync(kFull, mine.x, PARTS), __shfl_xor_sync(kFull, mine.y, PARTS),
                            __shfl_xor_sync(kFull, mine.z, PARTS));
    SurfaceShade o;
    if (lane == 0 && k < n) {
        if (ok) shade_from_lookups(s, L, dir, mine, other, &o);
        else shade_nothing(s.position, &o);
        rays_out[i] = make_float4(o.base.x, o.base.y, o.base.z, t);
    }
    const bool enqueue = lane == 0 && ok;
    const uint32_t qk = warp_append(enqueue, q.count);
    if (enqueue) {
        q.idx[qk] = i;
        q.pos[qk] = make_float4(o.position.x, o.position.y, o.position.z, 0.0f);
        q.sun[qk] = make_float4(o.sun.x, o.sun.y, o.sun.z, o.fade);
    }
}

struct BatchShadowJob {
    static constexpr float kTmin = 0.1f;
    static constexpr uint32_t kMask = 0xFFu;
    const ShadowQueue q;
    BatchTables bt;
    float4* rays;
    uint32_t* prim;

    template <class W>
    __device__ __forceinline__ bool start(W& w, const DeviceScene& sc, uint32_t id, uint32_t* out) const {
        *out = id;
        float4 p = q.pos[id];
        uint32_t v = __float_as_uint(p.w);
        if (v >= bt.nvol) {
            raise_error(bt.err, DEV_BAD_INDEX);
            v = 0;
        }
        const BatchVolume& vol = bt.vols[v];
        return w.start_at(sc, W::kWide ? vol.wroot : vol.root, f3(p.x, p.y, p.z),
                          f3(vol.L.dir[0], vol.L.dir[1], vol.L.dir[2]), 10000.0f);
    }
    template <class W>
    __device__ __forceinline__ void finish(const W& w, uint32_t id) const {
        uint32_t idx = q.idx[id];
        if (w.best.inst != kNoHit) {
            prim[idx] |= 1u << 30;
            return;
        }
        float4 sun = q.sun[id];
        float4 rec = rays[idx];
        float3 c = (f3(rec.x, rec.y, rec.z) + f3(sun.x, sun.y, sun.z)) * sun.w;
        rays[idx] = make_float4(c.x, c.y, c.z, rec.w);
    }
};

template <class Stack, template <bool, class> class Walker>
__global__ void __launch_bounds__(kPersistThreads, Walker<false, Stack>::kMinBlocks) k_batch_primary(DeviceScene arena, BatchPrimaryJob job,
                                                                   uint32_t total, uint32_t* counter, int stack_cap,
                                                                   int split, WalkKnobs knobs) {
    persistent_walk<false, Stack, Walker>(arena, job, total, counter, stack_cap, split, knobs, job.bt.err);
}

template <class Stack, template <bool, class> class Walker>
__global__ void __launch_bounds__(kPersistThreads, Walker<false, Stack>::kMinBlocks) k_batch_shadow(DeviceScene arena, BatchShadowJob job,
                                                                  const uint32_t* qcount, uint32_t* counter,
                                                                  int stack_cap, int split, WalkKnobs knobs) {
    persistent_walk<true, Stack, Walker>(arena, job, *qcount, counter, stack_cap, split, knobs, job.bt.err);
}

// Batched shading, pass 1 (k_shade_classify with the record's volume).
__global__ void __launch_bounds__(kClassifyThreads) k_batch_classify(BatchTables bt, uint32_t total, WaveHits hits,
                                                        float4* rays_out, uint32_t* front_count) {
    const uint32_t i = bt.first + blockIdx.x * blockDim.x + threadIdx.x;
    bool is_front = false;
    if (i < bt.first + total) {
        const float4 th = hits.thit[i];
        const uint32_t pb = hits.prim[i];
        const uint32_t inst = __float_as_uint(th.w);
        const bool back = (pb >> 31) != 0;
        if (inst == kNoHit) {
            const BatchVolume& vol = bt.vols[batch_volume(bt, i)];
            rays_out[i] = make_float4(vol.L.sky[0], vol.L.sky[1], vol.L.sky[2], -1.0f);
        } else if (back) {
            rays_out[i] = make_float4(0.0f, 0.0f, 0.0f, th.x * 0.80f);
        } else {
            is_front = true;
        }
    }
    const uint32_t k = block_append(is_front, front_count);
    if (is_front) hits.front[k] = i;
}

// Batched shading, pass 2 (k_shade_front with the volume's scene, grid,
// light, states and atlas; the shadow-queue entry carries the volume).
// Four resident blocks per SM (the volume's tables take registers that the
// other form has in constants): a twelve-volume update 5.88 ms against 5.95 ms
// at five and 6.00 ms at six.
__global__ void __launch_bounds__(128, 4) k_batch_shade_front(BatchTables bt, WaveHits hits,
                                                              const uint32_t* front_count, float4* rays_out,
                                                              ShadowQueue q) {
    const uint32_t n = *front_count;
    if (blockIdx.x * blockDim.x >= n) return;  // whole block
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    bool enqueue = false;
    SurfaceShade s;
    uint32_t i = 0, v = 0;
    if (k < n) {
        i = hits.front[k];
        v = batch_volume(bt, i);
        const BatchVolume& vol = bt.vols[v];
        const uint32_t R = vol.g.rays;
        const uint32_t local = i - __ldg(bt.ray_base + v);
        const uint32_t slot = local / R, ray = local - slot * R;
        const float4 th = hits.thit[i];
        const uint32_t inst = __float_as_uint(th.w), prim = hits.prim[i] & 0x0fffffffu;
        const float4 d4 = __ldg(bt.dirs + vol.dir_base + ray);
        const float3 d = f3(d4.x, d4.y, d4.z);
        const float3 o = probe_origin_exact(vol.g, slot);
        const bool half = vol.fp16 != 0;
        AtlasView<ColorTexDyn, DepthTexDyn> at{{vol.color, half}, {vol.depth, half}};
        enqueue = shade_surface(vol.sc, vol.g, vol.L, vol.states, at, o, d, th.x, th.y, th.z, inst, prim, &s, bt.err);
        rays_out[i] = make_float4(s.base.x, s.base.y, s.base.z, th.x);
    }
    const uint32_t qk = warp_append(enqueue, q.count);
    if (enqueue) {
        q.idx[qk] = i;
        q.pos[qk] = make_float4(s.position.x, s.position.y, s.position.z, __uint_as_float(v));
        q.sun[qk] = make_float4(s.sun.x, s.sun.y, s.sun.z, s.fade);
    }
}

// Shared memory of a block's stacks.
size_t walker_smem(int entries) { return (size_t)entries * kPersistThreads * sizeof(int); }

uint32_t persistent_blocks(const void* kernel, size_t smem, uint32_t cap_per_sm = 0) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kPersistThreads, smem);
    if (per <= 0) per = 1;
    if (cap_per_sm > 0 && (uint32_t)per > cap_per_sm) per = (int)cap_per_sm;
    return (uint32_t)(sms * per);
}

// Lanes per hit of the front-hit shading for at most `total` hits, from the
// threads resident at a time (`slots`, 97,280 on 152 SMs).  The kernel by itself
// in rooms of 128 rays a probe, all probes, 1 / 2 / 4 lanes (us):
//   records      32,768         65,536         98,304         196,608
//   FP32 atlas   21 / 13 / 13   25 / 17 / 23   28 / 31 / 34   60 / 46 / 62
//   FP16 atlas   18 / 13 / 12   19 / 16 / 21   21 / 26 / 28   43 / 41 / 54
// Four lanes win while they fit with the hits' usual share of the records, two
// while the launch fits in a round and a half; beyond that one lane over an FP16
// atlas.  Over an FP32 atlas, where one lane's two lookups spill registers, two
// lanes go on.  Whole updates, two lanes against one (300 boxes in a room; a
// terrain of 1,025 instances):
//   records   98,304  131,072  196,608  262,144  524,288  1.05 M  2.1 M   4.2 M
//   room      +2.1 %  0        -5.7 %   -0.7 %   -1.5 %   -2.4 %  -2.0 %  -1.5 %
//   terrain   -1.5 %  +0.1 %   +0.4 %   -2.8 %   -1.3 %   -0.4 %  -0.4 %  0
// They lose where one lane's threads fit in a round and two lanes' just do not,
// which depends on the hits' share of the records, so no line avoids it.  The
// largest launches are left to one lane: a terrain of 4,097 instances at 4.2 M
// records 6,333 against 6,389 us, its scheduled frame of 3.1 M 1,540 against 1,560.
uint32_t shade_lanes(uint32_t total, bool fp16_atlas) {
    const uint32_t slots = kShadeBlocksPerSm * 128u * sm_count();
    if (total <= slots / 3u) return 4u;
    return total <= (fp16_atlas ? slots / 4u * 3u : slots * 16u) ? 2u : 1u;
}

}  // namespace

namespace {

template <class Stack, template <bool, class> class Walker>
cudaError_t wavefront_kernels(const DeviceScene& sc, const DeviceGrid& g, const DeviceLight& L,
                              const uint32_t* probe_list, uint32_t total, const float4* dirs, const uint32_t* states,
                              const void* color, const void* depth, bool fp16_atlas, WaveHits hits, ShadowQueue q,
                              uint32_t* counters, float4* rays_out, ddgi_hit* hits_out, int stack_cap, int split,
                              uint32_t* err, cudaStream_t st, cudaEvent_t after_primary, const uint32_t* dev_count,
                              const TraceTuning& tune, const PrimaryJob& pj) {
    const size_t smem = walker_smem(split);
    const WalkKnobs knobs = walk_knobs(tune);
    k_primary<Stack, Walker><<<persistent_blocks((const void*)k_primary<Stack, Walker>, smem, tune.ctas_per_sm),
                               kPersistThreads, smem, st>>>(sc, pj, counters, stack_cap, split, knobs, err);
    if (after_primary) cudaEventRecord(after_primary, st);
    ShadowQueue qq = q;
    qq.count = counters + 1;
    cudaError_t e = launch_dependent(k_shade_classify, (total + kClassifyThreads - 1) / kClassifyThreads,
                                     kClassifyThreads, 0, st, g, L, total, hits, rays_out, hits_out,
                                     counters + 3, dev_count);
    if (e != cudaSuccess) return e;
    const uint32_t lanes = shade_lanes(total, fp16_atlas);
    const uint32_t shade_blocks = (uint32_t)(((uint64_t)total * lanes + 127) / 128);
    auto shade = [&](auto at) {
        auto launch = [&](auto kernel) {
            return launch_dependent(kernel, shade_blocks, 128, 0, st, sc, g, L, probe_list, dirs, states, at, hits,
                                    counters + 3, rays_out, qq, err);
        };
        if (lanes == 4u) return launch(k_shade_front_split<2, decltype(at)>);
        if (lanes == 2u) return launch(k_shade_front_split<1, decltype(at)>);
        return launch(k_shade_front<decltype(at)>);
    };
    e = fp16_atlas ? shade(AtlasView<ColorTexF16, DepthTexF16>{{static_cast<const uint2*>(color)},
                                                               {static_cast<const uint32_t*>(depth)}})
                   : shade(AtlasView<ColorTexF32, DepthTexF32>{{static_cast<const float4*>(color)},
                                                               {static_cast<const float2*>(depth)}});
    if (e != cudaSuccess) return e;
    ShadowJob sj{qq, make_float3(L.dir[0], L.dir[1], L.dir[2]), rays_out, hits.prim, 0};
    e = launch_dependent(k_shadow<Stack, Walker>,
                         persistent_blocks((const void*)k_shadow<Stack, Walker>, smem, tune.ctas_per_sm),
                         kPersistThreads, smem, st, sc, sj, counters + 1, counters + 2, stack_cap, split, knobs, err);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

cudaError_t launch_wavefront(const DeviceScene& sc, const DeviceGrid& g, const DeviceLight& L,
                             const uint32_t* probe_list, uint32_t nprobes, const float4* dirs,
                             const uint32_t* ray_order, const uint32_t* states, const void* color, const void* depth,
                             bool fp16_atlas, WaveHits hits, ShadowQueue q, uint32_t* counters, float4* rays_out,
                             ddgi_hit* hits_out, int stack_cap, int wstack_cap, uint32_t* err, cudaStream_t st,
                             cudaEvent_t after_primary, const uint32_t* dev_count, const TraceTuning& tune,
                             const uint32_t* perm) {
    uint32_t total = nprobes * g.rays;
    if (total == 0) return cudaSuccess;
    // counters[0]: primary work, [1]: shadow queue length, [2]: shadow work, [3]: front-hit queue length
    cudaError_t e = cudaMemsetAsync(counters, 0, 4 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t rpw = grouped_rays_per_warp(tune.rays_per_warp, g.rays);
    // the grouped order covers all probes in perm order: no list, no device count
    const uint32_t* pm = (perm && !probe_list && !dev_count && rpw != 0u) ? perm : nullptr;
    PrimaryJob pj{g, probe_list, dirs, ray_order, hits, total, dev_count, pm, rpw, nprobes};
    const bool wide = tune.wide && sc.wnodes && sc.winstances && wstack_cap > 0;
    const int cap = wide ? wstack_cap : stack_cap;
    const bool split = !(tune.split == 0 || (int)tune.split >= cap);
    const int sp = split ? (int)tune.split : cap;
#define DDGI_WAVE(STACK, WALKER)                                                                                       \
    return wavefront_kernels<STACK, WALKER>(sc, g, L, probe_list, total, dirs, states, color, depth, fp16_atlas, hits, \
                                            q, counters, rays_out, hits_out, cap, sp, err, st, after_primary,         \
                                            dev_count, tune, pj)
    if (wide) {
        if (split) DDGI_WAVE(SplitStack, WideWalker);
        DDGI_WAVE(SmemStack, WideWalker);
    }
    if (split) DDGI_WAVE(SplitStack, WarpWalker);
    DDGI_WAVE(SmemStack, WarpWalker);
#undef DDGI_WAVE
}

namespace {

template <class Stack, template <bool, class> class Walker>
cudaError_t batch_trace_kernels(const DeviceScene& arena, const BatchTables& bt, uint32_t total, WaveHits hits,
                                ShadowQueue q, uint32_t* counters, float4* rays_out, int stack_cap, int split,
                                const TraceTuning& tune, cudaStream_t st, cudaEvent_t after_primary,
                                cudaEvent_t after_shade) {
    const size_t smem = walker_smem(split);
    const WalkKnobs knobs = walk_knobs(tune);
    BatchPrimaryJob pj{bt, hits};
    k_batch_primary<Stack, Walker>
        <<<persistent_blocks((const void*)k_batch_primary<Stack, Walker>, smem, tune.ctas_per_sm), kPersistThreads,
           smem, st>>>(arena, pj, total, counters, stack_cap, split, knobs);
    if (after_primary) cudaEventRecord(after_primary, st);
    ShadowQueue qq = q;
    qq.count = counters + 1;
    k_batch_classify<<<(total + kClassifyThreads - 1) / kClassifyThreads, kClassifyThreads, 0, st>>>(bt, total, hits, rays_out, counters + 3);
    k_batch_shade_front<<<(total + 127) / 128, 128, 0, st>>>(bt, hits, counters + 3, rays_out, qq);
    if (after_shade) cudaEventRecord(after_shade, st);
    BatchShadowJob sj{qq, bt, rays_out, hits.prim};
    k_batch_shadow<Stack, Walker>
        <<<persistent_blocks((const void*)k_batch_shadow<Stack, Walker>, smem, tune.ctas_per_sm), kPersistThreads,
           smem, st>>>(arena, sj, counters + 1, counters + 2, stack_cap, split, knobs);
    return cudaGetLastError();
}

}  // namespace

// counters[0..3] (primary work, shadow queue length, shadow work, front-hit
// queue length) must be zero when the launch sequence starts.
cudaError_t launch_batch_trace(const DeviceScene& arena, const BatchTables& bt, uint32_t total, WaveHits hits,
                               ShadowQueue q, uint32_t* counters, float4* rays_out, int stack_cap, int wstack_cap,
                               const TraceTuning& tune, cudaStream_t st, cudaEvent_t after_primary,
                               cudaEvent_t after_shade) {
    if (total == 0) return cudaSuccess;
    const bool wide = tune.wide && arena.wnodes && arena.winstances && wstack_cap > 0;
    const int cap = wide ? wstack_cap : stack_cap;
    const bool split = !(tune.split == 0 || (int)tune.split >= cap);
    const int sp = split ? (int)tune.split : cap;
#define DDGI_BATCH(STACK, WALKER)                                                                            \
    return batch_trace_kernels<STACK, WALKER>(arena, bt, total, hits, q, counters, rays_out, cap, sp, tune, \
                                              st, after_primary, after_shade)
    if (wide) {
        if (split) DDGI_BATCH(SplitStack, WideWalker);
        DDGI_BATCH(SmemStack, WideWalker);
    }
    if (split) DDGI_BATCH(SplitStack, WarpWalker);
    DDGI_BATCH(SmemStack, WarpWalker);
#undef DDGI_BATCH
}

// Probe classification of all P probes into `states`.  `dirs` holds the
// kInitRays init directions; back/near are P-entry scratch arrays.
cudaError_t launch_init_probes(const DeviceScene& sc, const DeviceGrid& g, const float4* dirs, uint32_t P,
                               uint32_t* back, uint32_t* near, uint32_t* states, uint32_t* counters, int stack_cap,
                               uint32_t* err, cudaStream_t st) {
    if (P == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(back, 0, sizeof(uint32_t) * P, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(near, 0, sizeof(uint32_t) * P, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(counters, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const size_t smem = walker_smem(stack_cap);
    InitJob job{g, dirs, 1.5f * g.cell_len, back, near};
    k_init_probes<<<persistent_blocks((const void*)k_init_probes, smem), kPersistThreads, smem, st>>>(
        sc, job, P * kInitRays, counters, stack_cap, err);
    k_init_states<<<(P + 255) / 256, 256, 0, st>>>(P, g.rays, back, near, states);
    return cudaGetLastError();
}

}  // namespace ddgi
