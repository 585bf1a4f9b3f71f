// traverse.cuh — two-level LBVH traversal (closest hit and any hit).
//
// The top-level tree is walked in world space; at an instance leaf an EXIT
// marker is pushed, the ray moves into object space through the instance's
// world-to-object transform and the mesh tree is walked; popping the marker
// restores the world ray.  Hits are accepted for t in [tmin, tmax]; among
// equal t the lowest (instance, primitive) wins, so the result does not
// depend on the visiting order.
#pragma once

#include "common.cuh"

namespace ddgi {

constexpr int kStack = 64;
constexpr int kExit = 0x7fffffff;
constexpr int kNone = (int)0x80000000;  // no node (never a valid reference)
constexpr uint32_t kNoHit = 0xFFFFFFFFu;
// Box tests use [tmin * kBoxLo, tcur * kBoxHi]: a relative margin far above
// the few-ulp error of slab and triangle distances, so that pruning never
// removes a box holding a hit the triangle test reports, at any ray length.
constexpr float kBoxLo = 0.99999f;
constexpr float kBoxHi = 1.00001f;

struct HitRec {
    float t, b1, b2;
    uint32_t inst, prim;
    bool back;
};

// Fetch counters of the measurement variant (COUNT = true): inner nodes
// visited, triangles tested, instances entered, rays traced (index 0 for
// closest-hit rays, 1 for any-hit rays), and shading bytes.
struct Fetches {
    uint32_t nodes[2] = {0, 0}, tris[2] = {0, 0}, insts[2] = {0, 0}, rays[2] = {0, 0}, shade_bytes = 0;
    uint32_t top_nodes[2] = {0, 0};  // the part of `nodes` in the top-level tree
};

// Closest hit (ANY = false) or any hit (ANY = true) with t in [tmin, tmax];
// ties on t go to the lowest (instance, primitive).
template <bool ANY, bool COUNT = false>
__device__ __forceinline__ bool traverse(const DeviceScene& sc, float3 wo, float3 wd, float tmin, float tmax,
                                         uint32_t mask, HitRec* best, uint32_t* err, Fetches* fc = nullptr) {
    if (COUNT) fc->rays[ANY]++;
    best->inst = kNoHit;
    best->prim = 0;
    best->t = tmax;
    best->b1 = best->b2 = 0.0f;
    best->back = false;
    if (sc.tlas_root < 0) return false;
    Ray r;
    ray_setup(r, wo, wd);
    int stack[kStack];
    int sp = 0;
    int ref = sc.tlas_root;
    bool in_blas = false;
    uint32_t inst_id = 0;
    float tcur = tmax;
    // A well-formed tree visits each node at most once per ray; the cap only
    // stops a malformed one from looping.
    for (uint32_t steps = 0;; ++steps) {
        if (steps > 4u * (sc.node_count + sc.tri_count + sc.instance_count) + 64u) {
            raise_error(err, DEV_BAD_INDEX);
            return best->inst != kNoHit;
        }
        if (ref >= 0) {
            if (COUNT) {
                fc->nodes[ANY]++;
                if (!in_blas) fc->top_nodes[ANY]++;
            }
            if ((uint32_t)ref >= sc.node_count) {
                raise_error(err, DEV_BAD_INDEX);
                return best->inst != kNoHit;
            }
            BvhNode n = load_node(sc.nodes, ref);
            bool h0, h1;
            float t0, t1;
            node_hit(r, n, tmin * kBoxLo, tcur * kBoxHi, &h0, &h1, &t0, &t1);
            if (h0 && h1) {
                int nearr = n.d.x, farr = n.d.y;
                if (t1 < t0) {
                    nearr = n.d.y;
                    farr = n.d.x;
                }
                if (sp >= kStack) {
                    raise_error(err, DEV_STACK_OVERFLOW);
                    return best->inst != kNoHit;
                }
                stack[sp++] = farr;
                ref = nearr;
                continue;
            }
            if (h0) {
                ref = n.d.x;
                continue;
            }
            if (h1) {
                ref = n.d.y;
                continue;
            }
        } else if (!in_blas) {
            // top-level leaf: one instance
            if ((uint32_t)((~ref) >> 3) >= sc.instance_count) {
                raise_error(err, DEV_BAD_INDEX);
                return best->inst != kNoHit;
            }
            const GpuInstance* gi = sc.instances + ((~ref) >> 3);
            int4 meta = __ldg(reinterpret_cast<const int4*>(gi) + 3);  // blas_root, custom, mask, id
            if (((uint32_t)meta.z & mask) != 0 && meta.x >= 0) {
                if (COUNT) fc->insts[ANY]++;
                if (sp >= kStack) {
                    raise_error(err, DEV_STACK_OVERFLOW);
                    return best->inst != kNoHit;
                }
                stack[sp++] = kExit;
                float4 w[3] = {__ldg(&gi->w2o[0]), __ldg(&gi->w2o[1]), __ldg(&gi->w2o[2])};
                float3 oo, od;
                xform_exact(w, wo, wd, &oo, &od);
                ray_setup(r, oo, od);
                inst_id = (uint32_t)meta.w;
                in_blas = true;
                ref = meta.x;
                continue;
            }
        } else {
            int first = (~ref) >> 3, count = ((~ref) & 7) + 1;
            if ((uint32_t)first + (uint32_t)count > sc.tri_count) {
                raise_error(err, DEV_BAD_INDEX);
                return best->inst != kNoHit;
            }
            if (COUNT) fc->tris[ANY] += count;
            for (int k = 0; k < count; ++k) {
                const float4* tp = reinterpret_cast<const float4*>(sc.tris + first + k);
                float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                float t, b1, b2;
                bool back;
                if (tri_hit_exact(r, f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z), tmin, tcur, &t, &b1, &b2,
                                  &back)) {
                    uint32_t prim = (uint32_t)__float_as_int(a.w);
                    bool better = ANY || best->inst == kNoHit || t < best->t ||
                                  (t == best->t && (inst_id < best->inst || (inst_id == best->inst && prim < best->prim)));
                    if (better) {
                        best->t = t;
                        best->inst = inst_id;
                        best->prim = prim;
                        best->b1 = b1;
                        best->b2 = b2;
                        best->back = back;
                        tcur = t;
                        if (ANY) return true;
                    }
                }
            }
        }
        // pop
        for (;;) {
            if (sp == 0) return best->inst != kNoHit;
            ref = stack[--sp];
            if (ref != kExit) break;
            in_blas = false;
            ray_setup(r, wo, wd);
        }
    }
}


// Bound by instruction issue under divergence (12 of 32 threads an
// instruction, L2 latency behind it).  Primary rays of the 1M-triangle
// terrain (4.2 M): 6.41 ms and 5.73 G warp instructions with lower and upper
// planes, a vote and four branches a visit; 5.70 ms with boxes as centre and
// half extent, 256-bit node loads, packed tests and one pop for all ways out
// of a visit; 4.76 ms and 3.98 G with three visits a vote and leaves held by
// kind.  A small room's 65 K: 98 -> 59 us, its shadow rays 49 -> 31 us.
//
// Warp-cooperative traversal for persistent kernels (Aila & Laine 2009,
// "while-while" with postponed leaves): every lane of the warp calls
// advance() together.  In phase 1 lanes walk inner nodes; a lane that meets a
// leaf keeps it and goes on walking until every lane holds a leaf (or has
// run out of nodes), so inner-node iterations stay busy.  Phase 2 processes
// the held leaves: an instance leaf moves the ray into the mesh tree, a
// triangle leaf runs the watertight tests.  The stack lives in shared memory
// (one column per thread).  Hit set, tie rule and results equal `traverse`.
// Threads of the blocks that run the walkers: a thread's stack entry i is
// at column i * kWalkerThreads of the block's shared array.
constexpr int kWalkerThreads = 128;
struct SmemStack {
    int* base;
    __device__ __forceinline__ int get(int i) const { return base[i * kWalkerThreads]; }
    __device__ __forceinline__ void set(int i, int v) { base[i * kWalkerThreads] = v; }
};

// The first `split` entries in shared memory, deeper ones in a per-thread
// local-memory array (L1-cached).  A smaller shared-memory part lets more
// warps reside per SM; traversals deeper than `split` pay local accesses.
// The local part is an array of the caller's (kSpillMax entries), kept out of
// the walker so that the walker's own fields stay in registers.
constexpr int kSpillMax = 96;
struct SplitStack {
    int* base;
    int split;
    int* spill;
    __device__ __forceinline__ int get(int i) const { return i < split ? base[i * kWalkerThreads] : spill[i - split]; }
    __device__ __forceinline__ void set(int i, int v) {
        if (i < split) base[i * kWalkerThreads] = v;
        else spill[i - split] = v;
    }
};

// World-space origin and direction of a walk: the top level needs only the
// box ray besides them (its leaves are instances, never triangles), made again
// when the walk leaves a mesh tree, which keeps values out of the registers
// of the persistent kernels.
struct WorldRay {
    float3 o, d;
};

// A ray as the box tests use it: the negated origin, the reciprocals of the
// direction and their magnitudes, paired (x, y) and (z, z) for the packed
// instructions.  The reciprocal is the approximate one (1 ulp); box distances
// carry a margin for it (kSlab).
//
// A direction component below 2^-66 stands in as +-2^-66.  Over a distance t
// that moves the ray by at most 2^-66 t, within the 1e-7 by which every box is
// enlarged at least for t up to 7e12, where the triangle test's own products
// pass the largest float.  And a centre's distance times the reciprocal stays
// finite for every box that has a finite form (kWalkReach).
struct BoxRay {
    uint64_t oxy, ozz, ixy, izz, axy, azz;
    __device__ __forceinline__ void set(float3 o, float3 d) {
        const float x = rcp(d.x), y = rcp(d.y), z = rcp(d.z);
        oxy = pack2(-o.x, -o.y);
        ozz = pack2(-o.z, -o.z);
        ixy = pack2(x, y);
        izz = pack2(z, z);
        axy = pack2(fabsf(x), fabsf(y));
        azz = pack2(fabsf(z), fabsf(z));
    }
    __device__ __forceinline__ float3 negated_origin() const {
        float x, y, z, z2;
        unpack2(oxy, &x, &y);
        unpack2(ozz, &z, &z2);
        return f3(x, y, z);
    }
    static __device__ __forceinline__ float rcp(float v) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(copysignf(fmaxf(fabsf(v), 0x1p-66f), v)));
        return r;
    }
};

// A box [c - h, c + h] is entered at (c - o) / d - h / |d| and left at
// (c - o) / d + h / |d| along each axis: an addition and a product for the
// centre and one multiply-add for either plane, with no minimum or maximum to
// tell the planes apart, and two values per packed instruction (9 packed, 6
// scalar multiply-adds, 8 minima and maxima and 2 scalings for a node's two
// boxes, against 44 instructions for lower and upper planes).
//
// Rounding: a plane's distance is off by at most 3 x 2^-23 of the centre's
// distance, plus the reciprocal's 2^-23.  Seen from outside a box that is
// relative to the distance itself, and kSlab, which scales the exit distance
// before it is compared with the entry, covers it sixteen-fold; near or inside
// a box it is relative to the box's own extent, and the builders enlarge
// every box by 1e-5 of that, 84 times the error.  Range: |c| <= 2^60, and a
// product (c - o) / d that overflows (|c - o| >= 2^62, by BoxRay's 2^66) belongs
// to a box that starts beyond t = 2^127.  Boxes that reach further than 2^60 have
// an infinite extent about zero, which prunes nothing: the entry is -infinity
// and the exit +infinity, or NaN, which the minima and maxima pass over.  So a
// box that holds a hit is never missed.
constexpr float kSlab = 1.00001f;

// Both boxes of a node: hit or not, and whether the second comes first, by
// entry distance, or by exit distance when the entries are equal (both boxes
// hold the ray's start, common at the top levels).
struct NodeHit {
    bool h0, h1, swap;
    int ref0, ref1;
};
__device__ __forceinline__ NodeHit walk_node_hit(const WalkNode* p, const BoxRay& r, float tmin, float tmax) {
    uint64_t c0, c1, cz, ref, h0, h1, hz, unused;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(c0), "=l"(c1), "=l"(cz), "=l"(ref) : "l"(p));
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4 + 32];" : "=l"(h0), "=l"(h1), "=l"(hz), "=l"(unused) : "l"(p));
    c0 = mul2(add2(c0, r.oxy), r.ixy);
    c1 = mul2(add2(c1, r.oxy), r.ixy);
    cz = mul2(add2(cz, r.ozz), r.izz);
    float a[2], b[2], z[2], ax, ay, az, hx, hy, x, y;
    unpack2(fma2(h0, r.axy, c0), &a[0], &a[1]);
    unpack2(fma2(h1, r.axy, c1), &b[0], &b[1]);
    unpack2(fma2(hz, r.azz, cz), &z[0], &z[1]);
    const float f0 = fmin3(a[0], a[1], fminf(z[0], tmax)), f1 = fmin3(b[0], b[1], fminf(z[1], tmax));
    unpack2(r.axy, &ax, &ay);
    unpack2(r.azz, &az, &x);
    unpack2(h0, &hx, &hy);
    unpack2(c0, &x, &y);
    a[0] = fmaf(-hx, ax, x);
    a[1] = fmaf(-hy, ay, y);
    unpack2(h1, &hx, &hy);
    unpack2(c1, &x, &y);
    b[0] = fmaf(-hx, ax, x);
    b[1] = fmaf(-hy, ay, y);
    unpack2(hz, &hx, &hy);
    unpack2(cz, &x, &y);
    z[0] = fmaf(-hx, az, x);
    z[1] = fmaf(-hy, az, y);
    const float n0 = fmax3(a[0], a[1], fmaxf(z[0], tmin)), n1 = fmax3(b[0], b[1], fmaxf(z[1], tmin));
    NodeHit n;
    n.h0 = n0 <= f0 * kSlab;
    n.h1 = n1 <= f1 * kSlab;
    n.swap = n1 < n0 || (n1 == n0 && f1 < f0);
    n.ref0 = (int)(uint32_t)ref;
    n.ref1 = (int)(uint32_t)(ref >> 32);
    return n;
}

// tri_hit_exact with the ray's shear in object space kept as its axis of
// largest direction (kz) and whether the direction is negative there, which
// exchanges the other two axes in the reference's test: that changes the sign
// of every edge function, the determinant and the scaled distance alike, so
// their quotients have the same bits and only the facing is turned round.
struct ShearRay {
    float Sx, Sy, Sz;
    uint32_t axis;  // kz | negative << 2
    __device__ __forceinline__ void set(float3 d) {
        uint32_t kz = 0;
        if (fabsf(d.y) > fabsf(d.x)) kz = 1;
        if (fabsf(d.z) > fabsf(sel3(d, (int)kz))) kz = 2;
        const float3 k = rotate(d, kz);
        Sx = __fdiv_rn(k.x, k.z);
        Sy = __fdiv_rn(k.y, k.z);
        Sz = __fdiv_rn(1.0f, k.z);
        axis = kz | (k.z < 0.0f ? 4u : 0u);
    }
    // the axes (kz + 1, kz + 2, kz) of v
    static __device__ __forceinline__ float3 rotate(float3 v, uint32_t kz) {
        return f3(kz == 0u ? v.y : (kz == 1u ? v.z : v.x), kz == 0u ? v.z : (kz == 1u ? v.x : v.y),
                  kz == 0u ? v.x : (kz == 1u ? v.y : v.z));
    }
};
__device__ __forceinline__ bool tri_hit_shear(const ShearRay& s, float3 no, float3 v0, float3 v1, float3 v2, float tmin,
                                              float tmax, float* t_out, float* b1, float* b2, bool* back) {
    const uint32_t kz = s.axis & 3u;
    const float3 A = s.rotate(f3(__fadd_rn(v0.x, no.x), __fadd_rn(v0.y, no.y), __fadd_rn(v0.z, no.z)), kz);
    const float3 B = s.rotate(f3(__fadd_rn(v1.x, no.x), __fadd_rn(v1.y, no.y), __fadd_rn(v1.z, no.z)), kz);
    const float3 C = s.rotate(f3(__fadd_rn(v2.x, no.x), __fadd_rn(v2.y, no.y), __fadd_rn(v2.z, no.z)), kz);
    const float Ax = __fsub_rn(A.x, __fmul_rn(s.Sx, A.z)), Ay = __fsub_rn(A.y, __fmul_rn(s.Sy, A.z));
    const float Bx = __fsub_rn(B.x, __fmul_rn(s.Sx, B.z)), By = __fsub_rn(B.y, __fmul_rn(s.Sy, B.z));
    const float Cx = __fsub_rn(C.x, __fmul_rn(s.Sx, C.z)), Cy = __fsub_rn(C.y, __fmul_rn(s.Sy, C.z));
    const float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    const float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    const float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    // edge functions of mixed signs: outside (U, V, W are finite here)
    if (fmin3(U, V, W) < 0.0f && fmax3(U, V, W) > 0.0f) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    const float Az = __fmul_rn(s.Sz, A.z), Bz = __fmul_rn(s.Sz, B.z), Cz = __fmul_rn(s.Sz, C.z);
    const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    const float t = __fdiv_rn(T, det);
    if (!(t >= tmin && t <= tmax)) return false;
    *t_out = t;
    *b1 = __fdiv_rn(V, det);
    *b2 = __fdiv_rn(W, det);
    *back = (det < 0.0f) != ((s.axis & 4u) != 0u);
    return true;
}

// Node visits between two votes of the search loop.  A vote with its branch
// costs a quarter of a visit, and a lane that finds its leaf goes on walking
// anyway.  Primary rays of the 1M-triangle terrain: 5.60 ms with one visit,
// 4.77 with two, 4.73 with three, 5.25 with four (the unrolled visits then
// pass the 64 registers of eight blocks per SM).
constexpr int kVisitsPerVote = 3;
// Held leaves of the kind (instance or triangles) that fewer lanes hold wait
// until this many do, but for seven calls at most.  Same rays: 4.98 ms when
// both kinds run in every call, 4.75 at 8, 4.73 at 12, 4.73 at 16.
constexpr uint32_t kLeafKindMin = 12;

template <bool ANY, class Stack = SmemStack>
struct WarpWalker {
    static constexpr bool kWide = false;
    // resident 128-thread blocks per SM the kernels are built for; the blocks'
    // shared-memory stacks fill an SM's shared memory
    static constexpr int kMinBlocks = 8;
    WorldRay wr;  // world ray
    BoxRay box;   // current ray (world or object space)
    ShearRay shear;  // object space
    Stack stk;
    int sp, cap, ref;
    int leaf;        // held leaf (kNone: none)
    bool in_blas;
    bool searching, bad;
    uint32_t inst_id, steps, mask;
    uint32_t wait_max;  // lanes still searching that no longer hold the warp in the search loop
    float tmin;
    HitRec best;  // best.t: the nearest hit so far, or the ray's end

    __device__ __forceinline__ void clear() {  // no ray
        ref = leaf = kNone;
        in_blas = false;
        steps = 0;
        best.t = 0.0f;
        box.set(f3(0, 0, 0), f3(1, 1, 1));
    }

    __device__ __forceinline__ bool start(const DeviceScene& sc, float3 o, float3 d, float tmax) {
        return start_at(sc, sc.tlas_root, o, d, tmax);
    }
    // Start at an explicit top-level root (several scenes in one node arena).
    __device__ __forceinline__ bool start_at(const DeviceScene& sc, int32_t root, float3 o, float3 d, float tmax) {
        wr.o = o;
        wr.d = d;
        box.set(o, d);
        best.inst = kNoHit;
        best.prim = 0;
        best.t = tmax;
        best.b1 = best.b2 = 0.0f;
        best.back = false;
        leaf = kNone;
        stk.set(0, kExit);  // the bottom of the stack: nothing is popped below it
        sp = 1;
        in_blas = false;
        inst_id = 0;
        steps = 0;
        ref = root >= 0 ? root : kNone;
        return ref != kNone;
    }

    __device__ __forceinline__ bool push(int v, uint32_t* err) {
        if (sp >= cap) {
            raise_error(err, DEV_STACK_OVERFLOW);
            return false;
        }
        stk.set(sp++, v);
        return true;
    }
    // pop within the current tree level (stops at an EXIT marker)
    __device__ __forceinline__ void pop_level() {
        const int v = stk.get(sp - 1);
        sp -= v != kExit ? 1 : 0;
        ref = v != kExit ? v : kNone;
    }
    // pop across EXIT markers (restoring the world ray); false when empty
    __device__ __forceinline__ bool pop() {
        ref = stk.get(sp - 1);
        if (ref == kExit) {  // the mesh tree is done
            if (sp == 1) return false;
            in_blas = false;
            box.set(wr.o, wr.d);
            --sp;
            ref = stk.get(sp - 1);
            if (ref == kExit) return false;  // and so is the top level
        }
        --sp;
        return true;
    }

    // One step of a searching lane: visits a node, or takes a leaf and goes on
    // with the stack's top.  Errors (a bad reference, a full stack, too many
    // steps) only end the search here; advance() reports them.
    __device__ __forceinline__ void step(const DeviceScene& sc, float blo, float bhi) {
        bool next;  // go on with the stack's top
        if ((uint32_t)ref < sc.node_count) {
            const NodeHit n = walk_node_hit(sc.walk + ref, box, blo, bhi);
            ++steps;
            const bool second = n.h1 && (n.swap || !n.h0);
            next = !(n.h0 || n.h1);
            bad = sp >= cap || steps > sc.max_steps;
            if (n.h0 && n.h1 && !bad) {
                stk.set(sp, second ? n.ref0 : n.ref1);
                ++sp;
            }
            ref = second ? n.ref1 : n.ref0;
        } else {
            bad = ref >= 0;
            next = leaf == kNone;
            if (next) leaf = ref;  // postpone it and keep walking
            else searching = false;  // holding a leaf and at a second one
        }
        if (next) {
            pop_level();
            searching = ref != kNone;
        }
        if (bad) searching = false;
    }

    // All lanes call this (`calls`: how often the warp has); returns true when
    // an active lane's ray is finished.
    __device__ __forceinline__ bool advance(const DeviceScene& sc, uint32_t* err, bool active, uint32_t calls) {
        // every call counts as a step too: a ray that stopped making progress
        // (a malformed tree or a scheduling bug) ends with an error, not a hang
        ++steps;
        bad = false;
        // (a lane that holds a leaf and stands at a second one has nothing to search)
        searching = active && ref != kNone && (leaf == kNone || ref >= 0);
        const float blo = tmin * kBoxLo, bhi = best.t * kBoxHi;  // best.t is fixed until the leaf phase
        // step while more than `wait_max` lanes are still searching for a
        // leaf (lanes already holding one walk on speculatively), but at least
        // once when any is, so every searching lane makes progress in every
        // call; the stragglers carry on in the next call instead of holding
        // the whole warp in this loop
        for (uint32_t it = 0;; ++it) {
            const unsigned waiting = __ballot_sync(0xffffffffu, searching && leaf == kNone);
            if (waiting == 0u || (it > 0u && (uint32_t)__popc(waiting) <= wait_max)) break;
#pragma unroll
            for (int k = 0; k < kVisitsPerVote; ++k)
                if (searching) step(sc, blo, bhi);
        }
        // the leaf phase runs for the kind of leaf that more lanes hold; the
        // other kind's lanes keep theirs for a call in which enough do
        const uint32_t tris = __popc(__ballot_sync(0xffffffffu, active && leaf != kNone && in_blas));
        const uint32_t insts = __popc(__ballot_sync(0xffffffffu, active && leaf != kNone && !in_blas));
        const bool both = (calls & 7u) == 0u || min(tris, insts) >= kLeafKindMin;
        if (!active) return false;
        if (bad || steps > sc.max_steps) {
            raise_error(err, sp >= cap ? DEV_STACK_OVERFLOW : DEV_BAD_INDEX);
            return true;
        }
        if (leaf != kNone) {
            if (!in_blas && (both || insts >= tris)) {
                const uint32_t slot = (uint32_t)((~leaf) >> 3);
                leaf = kNone;
                if (slot >= sc.instance_count) {
                    raise_error(err, DEV_BAD_INDEX);
                    return true;
                }
                const GpuInstance* gi = sc.instances + slot;
                int4 meta = __ldg(reinterpret_cast<const int4*>(gi) + 3);  // blas_root, custom, mask, id
                if (((uint32_t)meta.z & mask) != 0 && meta.x >= 0) {
                    if (ref != kNone && !push(ref, err)) return true;
                    if (!push(kExit, err)) return true;
                    float4 w[3] = {__ldg(&gi->w2o[0]), __ldg(&gi->w2o[1]), __ldg(&gi->w2o[2])};
                    float3 oo, od;
                    xform_exact(w, wr.o, wr.d, &oo, &od);
                    box.set(oo, od);
                    shear.set(od);
                    inst_id = (uint32_t)meta.w;
                    in_blas = true;
                    ref = meta.x;
                    return false;
                }
            } else if (in_blas && (both || tris >= insts)) {
                int first = (~leaf) >> 3, count = ((~leaf) & 7) + 1;
                leaf = kNone;
                if ((uint32_t)first + (uint32_t)count > sc.tri_count) {
                    raise_error(err, DEV_BAD_INDEX);
                    return true;
                }
                const float3 no = box.negated_origin();
                for (int k = 0; k < count; ++k) {
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + first + k);
                    float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                    float t, b1, b2;
                    bool back;
                    if (tri_hit_shear(shear, no, f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z), tmin, best.t,
                                      &t, &b1, &b2, &back)) {
                        uint32_t prim = (uint32_t)__float_as_int(a.w);
                        bool better = ANY || best.inst == kNoHit || t < best.t ||
                                      (t == best.t && (inst_id < best.inst || (inst_id == best.inst && prim < best.prim)));
                        if (better) {
                            best.t = t;
                            best.inst = inst_id;
                            best.prim = prim;
                            best.b1 = b1;
                            best.b2 = b2;
                            best.back = back;
                            if (ANY) return true;
                        }
                    }
                }
            } else {
                --steps;  // a call spent waiting is none
                return false;
            }
        }
        if (ref == kNone && !pop()) return true;
        return false;
    }
};

// ---------------------------------------------------------------------------
// Eight-wide traversal over quantised WideNode trees: the walker of
// WarpWalker (while-while, postponed leaves, shared-memory stack, straggler
// exit) with node groups in place of single references (Ylitie, Karras &
// Laine 2017): the current group is a node and the mask of its children
// still to visit, in the ray's octant order; visiting a child takes the
// highest bit; an inner child's own children are box-tested at once (all
// eight slots, one mask) and the rest of the current group is pushed as one
// stack entry (node index << 8 | mask).  The slab test of slot k along an
// axis is fma(q_k, 2^e * inv, (o_node - o_ray) * inv) with q_k the near or
// far bound byte, the same kind of rounding as the binary step's
// (lo - o) * inv; with the quantised boxes enclosing the binary tree's
// enlarged boxes and the same interval margins, pruning stays conservative.
// Hit set, tie rule and results equal the binary traversal's.
// ---------------------------------------------------------------------------
// Float of an 8-bit integer (exact): its bits under the exponent of 2^23.
__device__ __forceinline__ float byte_float(uint32_t b) { return __uint_as_float(0x4B000000u | b) - 8388608.0f; }
// The same for byte i of w, the float's bits assembled by one byte permute.
__device__ __forceinline__ float byte_float_at(uint32_t w, int i) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)i)) - 8388608.0f;
}

template <bool ANY, class Stack = SmemStack>
struct WideWalker {
    static constexpr bool kWide = true;
    static constexpr int kMinBlocks = 7;
    WorldRay wr;  // world ray
    Ray r;        // current ray (world or object space)
    Stack stk;
    int sp, cap;
    int node;       // node of the current group (kNone: none)
    uint32_t gmask;  // its children still to visit, bit (slot ^ oct)
    uint32_t oct;    // octant of r.d: bit k set when the direction's component k is negative
    bool in_blas;
    uint32_t inst_id, steps, mask;
    uint32_t wait_max;
    float tmin, tcur;
    HitRec best;

    __device__ __forceinline__ void clear() {  // no ray
        node = kNone;
        gmask = 0;
    }

    __device__ __forceinline__ static uint32_t octant_of(float3 d) {
        return (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    }

    // Box tests of a node's eight slots; the mask bit of slot k is k ^ oct.
    __device__ __forceinline__ uint32_t test_children(const DeviceScene& sc, int n) const {
        const float4* p = reinterpret_cast<const float4*>(sc.wnodes + n);
        const float4 org = __ldg(p);
        const uint32_t eb = __float_as_uint(org.w);
        const float lo = tmin * kBoxLo, hi = tcur * kBoxHi;
        float tn[8], tf[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            tn[k] = lo;
            tf[k] = hi;
        }
#define DDGI_AXIS(A, O, INV, ORG)                                                                         \
    {                                                                                                     \
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(p + 1 + A));                                 \
        const float s = __uint_as_float(((eb >> (8 * A)) & 0xFFu) << 23) * INV;                           \
        const float b = (ORG - O) * INV;                                                                  \
        const bool pos = INV >= 0.0f;                                                                     \
        const uint32_t n0 = pos ? q.x : q.z, n1 = pos ? q.y : q.w, f0 = pos ? q.z : q.x, f1 = pos ? q.w : q.y; \
        _Pragma("unroll") for (int k = 0; k < 8; ++k) {                                                   \
            const uint32_t nw = k < 4 ? n0 : n1, fw = k < 4 ? f0 : f1;                                    \
            const float a = fmaf(byte_float_at(nw, k & 3), s, b);                                         \
            const float c = fmaf(byte_float_at(fw, k & 3), s, b);                                         \
            tn[k] = fmaxf(tn[k], a);                                                                      \
            tf[k] = fminf(tf[k], c);                                                                      \
        }                                                                                                 \
    }
        DDGI_AXIS(0, r.o.x, r.inv.x, org.x)
        DDGI_AXIS(1, r.o.y, r.inv.y, org.y)
        DDGI_AXIS(2, r.o.z, r.inv.z, org.z)
#undef DDGI_AXIS
        uint32_t m = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (tn[k] <= tf[k]) m |= 1u << ((uint32_t)k ^ oct);
        return m;
    }

    __device__ __forceinline__ bool start(const DeviceScene& sc, float3 o, float3 d, float tmax) {
        return start_at(sc, sc.wtlas_root, o, d, tmax);
    }
    __device__ __forceinline__ bool start_at(const DeviceScene& sc, int32_t root, float3 o, float3 d, float tmax) {
        wr.o = o;
        wr.d = d;
        ray_setup(r, o, d);
        oct = octant_of(d);
        tcur = tmax;
        best.inst = kNoHit;
        best.prim = 0;
        best.t = tmax;
        best.b1 = best.b2 = 0.0f;
        best.back = false;
        sp = 0;
        in_blas = false;
        inst_id = 0;
        steps = 0;
        node = kNone;
        gmask = 0;
        if (root < 0 || (uint32_t)root >= sc.wnode_count) return false;
        node = root;
        gmask = test_children(sc, root);
        return gmask != 0;
    }
    __device__ __forceinline__ bool push(int v, uint32_t* err) {
        if (sp >= cap) {
            raise_error(err, DEV_STACK_OVERFLOW);
            return false;
        }
        stk.set(sp++, v);
        return true;
    }
    // next group within the current tree level (stops at an EXIT marker)
    __device__ __forceinline__ void pop_level() {
        if (sp == 0 || stk.get(sp - 1) == kExit) {
            node = kNone;
            gmask = 0;
            return;
        }
        const int e = stk.get(--sp);
        node = e >> 8;
        gmask = (uint32_t)e & 0xFFu;
    }
    // next group across EXIT markers (restoring the world ray); false when empty
    __device__ __forceinline__ bool pop() {
        for (;;) {
            if (sp == 0) return false;
            const int e = stk.get(--sp);
            if (e != kExit) {
                node = e >> 8;
                gmask = (uint32_t)e & 0xFFu;
                return true;
            }
            in_blas = false;
            r.o = wr.o;  // back at the top level
            r.d = wr.d;
            r.inv = ray_inv(r.d);
            oct = octant_of(r.d);
        }
    }
    __device__ __forceinline__ int child_ref(const DeviceScene& sc, int n, uint32_t slot) const {
        return __ldg(reinterpret_cast<const int*>(sc.wnodes + n) + 16 + slot);
    }

    // All lanes call this; returns true when an active lane's ray is finished.
    __device__ __forceinline__ bool advance(const DeviceScene& sc, uint32_t* err, bool active, uint32_t) {
        int leaf = kNone;
        bool failed = false;
        if (active && ++steps > sc.wmax_steps) {  // as in WarpWalker::advance
            raise_error(err, DEV_BAD_INDEX);
            failed = true;
        }
        bool searching = active && node != kNone && !failed;
        for (uint32_t it = 0;; ++it) {  // as in WarpWalker::advance
            const unsigned waiting = __ballot_sync(0xffffffffu, searching && leaf == kNone);
            if (waiting == 0u || (it > 0u && (uint32_t)__popc(waiting) <= wait_max)) break;
            if (searching) {
                if (gmask != 0u) {
                    const uint32_t key = 31u - (uint32_t)__clz(gmask);
                    const int c = child_ref(sc, node, key ^ oct);
                    if (c >= 0) {
                        if (++steps > sc.wmax_steps || (uint32_t)c >= sc.wnode_count) {
                            raise_error(err, DEV_BAD_INDEX);
                            failed = true;
                            searching = false;
                        } else {
                            gmask &= ~(1u << key);
                            const uint32_t m = test_children(sc, c);
                            if (m != 0u) {
                                if (gmask != 0u && !push((node << 8) | (int)gmask, err)) {
                                    failed = true;
                                    searching = false;
                                }
                                node = c;
                                gmask = m;
                            }
                        }
                    } else if (leaf == kNone) {
                        gmask &= ~(1u << key);
                        leaf = c;  // postpone it and keep walking
                    } else {
                        searching = false;  // holding a leaf and at a second one (it stays in the mask)
                    }
                } else {
                    pop_level();
                }
                if (searching && node == kNone) searching = false;
            }
        }
        if (!active) return false;
        if (failed) return true;
        if (leaf != kNone) {
            if (!in_blas) {
                uint32_t slot = (uint32_t)((~leaf) >> 3);
                if (slot >= sc.instance_count) {
                    raise_error(err, DEV_BAD_INDEX);
                    return true;
                }
                const GpuInstance* gi = sc.winstances + slot;
                int4 meta = __ldg(reinterpret_cast<const int4*>(gi) + 3);  // blas_root (wide), custom, mask, id
                if (((uint32_t)meta.z & mask) != 0 && meta.x >= 0) {
                    if ((uint32_t)meta.x >= sc.wnode_count) {
                        raise_error(err, DEV_BAD_INDEX);
                        return true;
                    }
                    if (node != kNone && gmask != 0u && !push((node << 8) | (int)gmask, err)) return true;
                    if (!push(kExit, err)) return true;
                    float4 w[3] = {__ldg(&gi->w2o[0]), __ldg(&gi->w2o[1]), __ldg(&gi->w2o[2])};
                    float3 oo, od;
                    xform_exact(w, wr.o, wr.d, &oo, &od);
                    ray_setup(r, oo, od);
                    oct = octant_of(od);
                    inst_id = (uint32_t)meta.w;
                    in_blas = true;
                    node = meta.x;
                    gmask = test_children(sc, meta.x);
                    if (gmask != 0u) return false;
                    node = kNone;  // the mesh tree's root misses: back up
                }
            } else {
                int first = (~leaf) >> 3, count = ((~leaf) & 7) + 1;
                if ((uint32_t)first + (uint32_t)count > sc.tri_count) {
                    raise_error(err, DEV_BAD_INDEX);
                    return true;
                }
                for (int k = 0; k < count; ++k) {
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + first + k);
                    float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                    float t, b1, b2;
                    bool back;
                    if (tri_hit_exact(r, f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z), tmin, tcur, &t, &b1,
                                      &b2, &back)) {
                        uint32_t prim = (uint32_t)__float_as_int(a.w);
                        bool better = ANY || best.inst == kNoHit || t < best.t ||
                                      (t == best.t && (inst_id < best.inst || (inst_id == best.inst && prim < best.prim)));
                        if (better) {
                            best.t = t;
                            best.inst = inst_id;
                            best.prim = prim;
                            best.b1 = b1;
                            best.b2 = b2;
                            best.back = back;
                            tcur = t;
                            if (ANY) return true;
                        }
                    }
                }
            }
        }
        if ((node == kNone || gmask == 0u) && !pop()) return true;
        return false;
    }
};

}  // namespace ddgi
