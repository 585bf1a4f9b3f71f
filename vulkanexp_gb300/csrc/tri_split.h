// tri_split.h — conservative bounds of the parts of a triangle on either
// side of a plane perpendicular to one axis: the reference split of the
// spatial-split tree builders, the host one (sbvh.cu) and the device one
// (gbuild.cu), which evaluate exactly these float operations and so produce
// the same trees.
//
// The part of a triangle T on one side of a plane is the convex hull of T's
// vertices on that side and the crossings of T's edges with the plane (the
// reference split of Stich, Friedrich & Dietrich 2009, "Spatial splits in
// bounding volume hierarchies", as in Embree's SBVH builder).  A crossing
// p + t (q - p), t = (pl - p_k) / (q_k - p_k), is evaluated from the
// triangle's own float vertices with interval arithmetic: every operation
// rounded to nearest and then widened by one ulp on each side (nextafterf),
// which contains the exact result; t is clamped to [0, 1], and the
// crossing's own axis is the plane exactly.  The boxes therefore contain
// the exact parts and are wider by a few ulps of the coordinates only.  A
// builder intersects them with the reference's box (which bounds the
// triangle's part inside earlier split planes), which keeps them
// conservative: the part of T inside the reference and below a plane lies
// in box(T below the plane) and in the reference's box; the part between
// two planes lies in box(T above the lower one) and box(T below the upper
// one).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "../../include/ddgi_exact.h"

namespace ddgi {

DDGI_HD static inline float ts_add(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
DDGI_HD static inline float ts_sub(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
DDGI_HD static inline float ts_mul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
DDGI_HD static inline float ts_div(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdiv_rn(a, b);
#else
    return a / b;
#endif
}
DDGI_HD static inline int32_t ts_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_int(x);
#else
    int32_t i;
    memcpy(&i, &x, 4);
    return i;
#endif
}
DDGI_HD static inline float ts_float(int32_t i) {
#ifdef __CUDA_ARCH__
    return __int_as_float(i);
#else
    float x;
    memcpy(&x, &i, 4);
    return x;
#endif
}
// The neighbouring float above / below x (nextafterf).  Floats of one sign are
// ordered as their bit patterns are, so the neighbour is the pattern one away;
// adding +0 makes one zero of the two, and +infinity is its own neighbour.
DDGI_HD static inline float ts_up(float x) {
    const int32_t i = ts_bits(ts_add(x, 0.0f)), s = i >> 31, j = i + s + s + 1;
    return ts_float(j < 0x7F800000 ? j : 0x7F800000);
}
DDGI_HD static inline float ts_down(float x) { return -ts_up(-x); }

DDGI_HD static inline bool ts_crosses(float p, float q, float pl) { return (p < pl && q > pl) || (p > pl && q < pl); }

// The crossing of edge p -> q with the plane x_K = pl, strictly between p and
// q: its bounds, added to lo/hi.  t = (pl - p_K) / (q_K - p_K) lies in (0, 1);
// numerator and denominator have the same sign, and rounding is monotonic, so
// of the four quotients of their intervals' ends the lowest is that of the
// smallest numerator and the largest denominator (magnitudes) and the highest
// the other way round, and of the four products of (q_a - p_a) and t, t >= 0,
// the signs tell the lowest and the highest.
template <int K>
DDGI_HD static inline void ts_crossing(const float* p, const float* q, float pl, float lo[3], float hi[3]) {
    // magnitudes: the interval's ends are the patterns one below and one above
    const int32_t n = ts_bits(fabsf(ts_sub(pl, p[K]))), d = ts_bits(fabsf(ts_sub(q[K], p[K])));
    float t0 = 0.0f, t1 = 1.0f;
    if (d > 1) {
        const float nhi = ts_float(n < 0x7F800000 ? n + 1 : n), dhi = ts_float(d < 0x7F800000 ? d + 1 : d);
        const int32_t c0 = ts_bits(ts_div(ts_float(n - 1), dhi)) - 1;
        t0 = ts_float(c0 > 0 ? c0 : 0);
        t1 = fminf(1.0f, ts_up(ts_div(nhi, ts_float(d - 1))));
    }
    lo[K] = hi[K] = pl;  // the crossing's own axis is the plane exactly
    for (int a = 0; a < 3; ++a) {
        if (a == K) continue;
        const float dd = ts_sub(q[a], p[a]);
        const float ddlo = ts_down(dd), ddhi = ts_up(dd);
        lo[a] = fminf(lo[a], ts_down(ts_add(p[a], ts_down(ts_mul(ddlo, ddlo >= 0.0f ? t0 : t1)))));
        hi[a] = fmaxf(hi[a], ts_up(ts_add(p[a], ts_up(ts_mul(ddhi, ddhi >= 0.0f ? t1 : t0)))));
    }
}

// Bounds of the parts of triangle `tri` (9 floats: v0, v1, v2) on either
// side of the plane x_K = pl: below (x_K <= pl) into llo/lhi, above
// (x_K >= pl) into glo/ghi.  A side the triangle misses stays empty (lo
// +inf, hi -inf).  K is a template argument so that a device caller keeps
// the triangle in registers.
template <int K>
DDGI_HD static inline void tri_plane_bounds_k(const float* tri, float pl, float llo[3], float lhi[3], float glo[3],
                                              float ghi[3]) {
    for (int a = 0; a < 3; ++a) {
        llo[a] = glo[a] = INFINITY;
        lhi[a] = ghi[a] = -INFINITY;
    }
    for (int v = 0; v < 3; ++v) {
        const float* p = tri + 3 * v;
        if (p[K] <= pl)
            for (int a = 0; a < 3; ++a) {
                llo[a] = fminf(llo[a], p[a]);
                lhi[a] = fmaxf(lhi[a], p[a]);
            }
        if (p[K] >= pl)
            for (int a = 0; a < 3; ++a) {
                glo[a] = fminf(glo[a], p[a]);
                ghi[a] = fmaxf(ghi[a], p[a]);
            }
    }
    // at most two edges cross: those of the vertex alone on its side
    const bool c0 = ts_crosses(tri[K], tri[3 + K], pl), c1 = ts_crosses(tri[3 + K], tri[6 + K], pl),
               c2 = ts_crosses(tri[6 + K], tri[K], pl);
    const int v = c0 ? (c1 ? 1 : 0) : (c1 && !c2 ? 1 : 2);
    float at[3], next[3], before[3];
    for (int a = 0; a < 3; ++a) {
        at[a] = v == 0 ? tri[a] : (v == 1 ? tri[3 + a] : tri[6 + a]);
        next[a] = v == 0 ? tri[3 + a] : (v == 1 ? tri[6 + a] : tri[a]);
        before[a] = v == 0 ? tri[6 + a] : (v == 1 ? tri[a] : tri[3 + a]);
    }
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    if (v == 0 ? c0 : (v == 1 ? c1 : c2)) ts_crossing<K>(at, next, pl, lo, hi);
    if (v == 0 ? c2 : (v == 1 ? c0 : c1)) ts_crossing<K>(before, at, pl, lo, hi);
    for (int a = 0; a < 3; ++a) {  // the crossings bound both sides
        llo[a] = fminf(llo[a], lo[a]);
        lhi[a] = fmaxf(lhi[a], hi[a]);
        glo[a] = fminf(glo[a], lo[a]);
        ghi[a] = fmaxf(ghi[a], hi[a]);
    }
}

DDGI_HD static inline void tri_plane_bounds(const float* tri, int k, float pl, float llo[3], float lhi[3], float glo[3],
                                            float ghi[3]) {
    if (k == 0) tri_plane_bounds_k<0>(tri, pl, llo, lhi, glo, ghi);
    else if (k == 1) tri_plane_bounds_k<1>(tri, pl, llo, lhi, glo, ghi);
    else tri_plane_bounds_k<2>(tri, pl, llo, lhi, glo, ghi);
}

// A reference box bounding the triangle's part inside `slab` (a reference's
// box with axis k narrowed to [slab_lo[k], slab_hi[k]]): the slab
// intersected with the triangle's bounds above slab_lo[k] and below
// slab_hi[k].  lo > hi in some axis when that leaves nothing.
DDGI_HD static inline void tri_split_box(const float* tri, int k, const float slab_lo[3], const float slab_hi[3],
                                         float out_lo[3], float out_hi[3]) {
    float llo[3], lhi[3], glo[3], ghi[3];
    for (int a = 0; a < 3; ++a) {
        out_lo[a] = slab_lo[a];
        out_hi[a] = slab_hi[a];
    }
    tri_plane_bounds(tri, k, slab_lo[k], llo, lhi, glo, ghi);
    for (int a = 0; a < 3; ++a) {
        out_lo[a] = fmaxf(out_lo[a], glo[a]);
        out_hi[a] = fminf(out_hi[a], ghi[a]);
    }
    tri_plane_bounds(tri, k, slab_hi[k], llo, lhi, glo, ghi);
    for (int a = 0; a < 3; ++a) {
        out_lo[a] = fmaxf(out_lo[a], llo[a]);
        out_hi[a] = fminf(out_hi[a], lhi[a]);
    }
}

}  // namespace ddgi
