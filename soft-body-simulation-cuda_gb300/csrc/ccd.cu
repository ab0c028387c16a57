// Continuous collision between bodies on the GPU (see ccd.h).
//
// The triangles stand in a fixed order, body after body and along each body's
// Morton curve at rest (build_ccd_surface): 32 in a row are a group, 32 groups
// a node above them, and so on.  The candidates do not depend on the tree, so
// a detection only computes its boxes:
//   1. k_boxes: swept box of every surface triangle (X -> XTilde), of every
//      group and of every 32 groups (k_boxes_up: what is above);
//   2. k_groups: a warp a group, 32 boxes a step down the tree: the pairs of
//      groups whose boxes overlap;
//   3. k_pairs: a warp a pair of groups: its triangles of different bodies that
//      share no vertex and whose boxes overlap (pairs kept once);
//   4. k_narrow: per pair and direction 3 point-face and 9 edge-edge
//      continuous tests; per vertex (point-face) and per edge (edge-edge)
//      the earliest contact before t = 1 by a 64-bit atomic minimum of
//      (contact time bits, face / other edge index);
//   5. k_mark, k_result: tI = 0.5 and the earliest touching contact's normal for
//      the vertices of every such contact (the reference's storeTi rule with its
//      write race replaced by the earliest-contact choice).
// Counts stay on the device; the host reads them once, at the end, and runs the
// detection again with larger lists when one was too short.
// What bounds a detection of some thousand triangles is latency: each kernel is
// a chain of a few loads.  A binary tree over Morton codes sorted anew each time
// (radix sort, build, refit, a stack a thread) took 240 us for 8 bodies of
// 6 to 12 cells a side.
// The reference's candidate set is the same (its BVH traversal is exact);
// its query and reduction semantics are restated in narrow_test() below
// (intersections.cu:286-334, narrowphase.cu:8-127).
//
// This unit is compiled without floating-point contraction, so the narrow
// phase performs the same IEEE single-precision operations as the CPU
// oracle and the reference's code compiled for the host.
#include "ccd.h"

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <utility>

#include "pdl.cuh"
#include "scene.cuh"

namespace pdgb {

namespace {

constexpr unsigned long long kNone = ~0ull;
constexpr int kThreads = 256;
constexpr int kBoxThreads = 1024;  // 32 groups of 32 triangles
constexpr unsigned int kMostPairs = 1u << 30;
// CTAs of the kernels that go over a list whose length is on the device: 4 on an
// SM, the fewest that their registers allow.
constexpr int kListCtas = 4 * 152;
constexpr int kMaxLevels = 7;      // 32^7 > 2^31 triangles
constexpr int kCounters = 4;

inline int blocks_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

// ------------------------------------------------------------ geometry
struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(float4 a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 scl(float s, F3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 cross(F3 a, F3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float len(F3 a) { return sqrtf(dot(a, a)); }
__device__ __forceinline__ F3 unit(F3 a) { return scl(1.0f / len(a), a); }
__device__ __forceinline__ float triple(F3 u, F3 v, F3 w) { return dot(u, cross(v, w)); }

// The query's thresholds are double literals in the reference.  FP64 compares
// in the Newton loop took most of the narrow phase (a conversion and a compare
// per iteration at two lanes a clock and SM), so they are decided in float:
// for a float f and a double threshold, f < 1e-6 holds exactly when
// f <= 1e-6f, the largest float below 1e-6, and so on.
constexpr float kBelow6 = 1e-6f;            // f < 1e-6   <=>  f <= kBelow6
constexpr float kUpTo3 = 0.00099999993f;    // f >= -1e-3 <=>  f >= -kUpTo3
constexpr float kBelow12 = 1e-12f;          // f < -1e-12 <=>  f < -kBelow12
static_assert((double)kBelow6 < 1e-6 && (double)kBelow6 * (1.0 + 1.2e-7) > 1e-6, "largest float below 1e-6");
static_assert((double)kUpTo3 <= 1e-3 && (double)kUpTo3 * (1.0 + 1.2e-7) > 1e-3, "largest float up to 1e-3");
static_assert((double)kBelow12 < 1e-12 && (double)kBelow12 * (1.0 + 1.2e-7) > 1e-12, "largest float below 1e-12");

// a > 1e-12 b in double (a, b >= 0): decided in float where the two differ by
// more than float's rounding, in double where they do not or could underflow.
__device__ __forceinline__ bool above_scaled(float a, float b) {
    if (b > 1e-20f && b < 1e30f) {
        if (a > 1.00001e-12f * b) return true;
        if (a < 0.99999e-12f * b) return false;
    }
    return a > 1e-12 * b;
}

// Real roots of a x^2 + b x + c in the numerically stable form; 0 with the
// vertex -b / 2a in x[0] when the discriminant is negative.
__device__ int quad_roots(float a, float b, float c, float* x) {
    const float d = b * b - 4 * a * c;
    if (d < 0) {
        x[0] = -b / (2 * a);
        return 0;
    }
    const float sgn = (b > 0) ? 1.0f : (b < 0 ? -1.0f : 0.0f);
    const float q = -(b + sgn * sqrtf(d)) / 2;
    int n = 0;
    if (above_scaled(fabsf(a), fabsf(q))) x[n++] = q / a;
    if (above_scaled(fabsf(q), fabsf(c))) x[n++] = c / q;
    if (n == 2 && x[0] > x[1]) {
        const float t = x[0];
        x[0] = x[1];
        x[1] = t;
    }
    return n;
}

// Newton iteration on the cubic from x0 (at most 100 steps); with dir != 0
// the start is first moved off the critical point by the quadratic model.
__device__ float cubic_newton(float a, float b, float c, float d, float x0, int dir) {
    if (dir != 0) {
        const float y0 = d + x0 * (c + x0 * (b + x0 * a));
        const float ddy0 = 2 * b + x0 * (6 * a);
        if (ddy0 != 0) x0 += dir * sqrtf(fabsf(2 * y0 / ddy0));
    }
    // Far roots and roots of near-planar queries end up going round a few floats
    // more than 1e-6 apart, mostly two, for the rest of the hundred steps.  A step
    // depends on the iterate alone, so once one repeats (Brent's cycle finding: the
    // iterates 2, 4, 8, .. are kept) whole rounds are left out.  8 bodies in
    // contact, where one query of sixty took 100 or 200 steps and its warp with
    // it: 62 -> 34 us (31 with the runs dealt out, k_narrow()).
    float kept = __int_as_float(0x7fffffff);  // NaN: none
    int kept_at = 0, next = 2, steps = 100;
    for (int it = 1; it <= steps; ++it) {
        const float y = d + x0 * (c + x0 * (b + x0 * a));
        const float dy = c + x0 * (2 * b + x0 * 3 * a);
        if (dy == 0) return x0;
        const float x1 = x0 - y / dy;
        if (fabsf(x0 - x1) <= kBelow6) return x0;
        if (x1 == kept) steps = it + (steps - it) % (it - kept_at);
        if (it == next) {
            kept = x1;
            kept_at = it;
            next *= 2;
        }
        x0 = x1;
    }
    return x0;
}

// Real roots of a x^3 + b x^2 + c x + d, bracketed by the critical points.
__device__ int cubic_roots(float a, float b, float c, float d, float* x) {
    float xc[2];
    const int ncrit = quad_roots(3 * a, 2 * b, c, xc);
    if (ncrit == 0) {
        x[0] = cubic_newton(a, b, c, d, xc[0], 0);
        return 1;
    }
    if (ncrit == 1) return quad_roots(b, c, d, x);
    const float yc0 = d + xc[0] * (c + xc[0] * (b + xc[0] * a));
    const float yc1 = d + xc[1] * (c + xc[1] * (b + xc[1] * a));
    int n = 0;
    if (yc0 * a >= 0) x[n++] = cubic_newton(a, b, c, d, xc[0], -1);
    if (yc0 * yc1 <= 0) {
        const int closer = fabsf(yc0) < fabsf(yc1) ? 0 : 1;
        x[n++] = cubic_newton(a, b, c, d, xc[closer], closer == 0 ? 1 : -1);
    }
    if (yc1 * a <= 0) x[n++] = cubic_newton(a, b, c, d, xc[1], 1);
    return n;
}

// Signed distance of p to the plane of face (y0, y1, y2), its normal and
// the barycentric weights (w0 = 1, w1..3 = minus the face coordinates).
__device__ float face_distance(F3 p, F3 y0, F3 y1, F3 y2, F3& n, float w[4]) {
    n = cross(unit(sub(y1, y0)), unit(sub(y2, y0)));
    if (dot(n, n) <= kBelow6) return FLT_MAX;
    n = unit(n);
    const float h = dot(sub(p, y0), n);
    const float b0 = triple(sub(y1, p), sub(y2, p), n), b1 = triple(sub(y2, p), sub(y0, p), n),
                b2 = triple(sub(y0, p), sub(y1, p), n);
    const float s = b0 + b1 + b2;
    w[0] = 1;
    w[1] = -b0 / s;
    w[2] = -b1 / s;
    w[3] = -b2 / s;
    return h;
}

// Signed distance between the lines of edges (x0, x1) and (y0, y1), their
// common normal and the weights (w0, w1 on the first, -w2, -w3 on the second).
__device__ float edge_distance(F3 x0, F3 x1, F3 y0, F3 y1, F3& n, float w[4]) {
    n = cross(unit(sub(x1, x0)), unit(sub(y1, y0)));
    if (dot(n, n) <= kBelow6) return FLT_MAX;
    n = unit(n);
    const float h = dot(sub(x0, y0), n);
    const float a0 = triple(sub(y1, x1), sub(y0, x1), n), a1 = triple(sub(y0, x0), sub(y1, x0), n);
    const float b0 = triple(sub(x0, y1), sub(x1, y1), n), b1 = triple(sub(x1, y0), sub(x0, y0), n);
    w[0] = a0 / (a0 + a1);
    w[1] = a1 / (a0 + a1);
    w[2] = -b0 / (b0 + b1);
    w[3] = -b1 / (b0 + b1);
    return h;
}

// a < 1e-12 l0 l1 l2 in double: decided in float where it is clear.
__device__ __forceinline__ bool coplanar(float a, float l0, float l1, float l2) {
    const float p = l0 * l1 * l2;
    if (p > 1e-20f && p < 1e30f) {
        if (a < 0.99999e-12f * p) return true;
        if (a > 1.00001e-12f * p) return false;
    }
    return a < 1e-12 * l0 * l1 * l2;
}

// Coplanarity cubic a[3] t^3 + .. + a[0] of four points x + t v: their signed
// volume at t.
__device__ __forceinline__ void volume_cubic(const F3 x[4], const F3 v[4], float a[4], F3& x01, F3& x02, F3& x03) {
    x01 = sub(x[1], x[0]), x02 = sub(x[2], x[0]), x03 = sub(x[3], x[0]);
    const F3 v01 = sub(v[1], v[0]), v02 = sub(v[2], v[0]), v03 = sub(v[3], v[0]);
    a[0] = triple(x01, x02, x03);
    a[1] = triple(v01, x02, x03) + triple(x01, v02, x03) + triple(x01, x02, v03);
    a[2] = triple(x01, v02, v03) + triple(v01, x02, v03) + triple(v01, v02, x03);
    a[3] = triple(v01, v02, v03);
}

__device__ __forceinline__ float abs_sum(F3 a) { return fabsf(a.x) + fabsf(a.y) + fabsf(a.z); }
__device__ __forceinline__ float abs_max(F3 a) { return fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))); }

// False where narrow_test() returns 1 for certain, without its Newton
// iterations (nine of ten candidates' queries): coplanar at t = 0, or a volume
// that stays away from zero.  On [0, 1] the cubic lies between the least and the
// greatest of its Bernstein coefficients.  A contact has a computed distance of
// at most 1e-6, and distance times the product of two edges (each at most 2 L,
// L the largest |x0k| + |v0k|) times the sine of their angle is the volume:
// 4e-6 L^2 at most.  Rounding moves the volume and the distance's normal by some
// tens of units in the last place of L^3 and of C L^2 (C the largest
// coordinate; the normal's error grows with the sine's inverse and cancels it).
// The line lies at 2e-5 L^2 + 4e-5 L^2 (C + L), 330 units; NaN is kept.
__device__ __forceinline__ bool may_touch(const F3 x[4], const F3 v[4]) {
    float a[4];
    F3 x01, x02, x03;
    volume_cubic(x, v, a, x01, x02, x03);
    if (coplanar(fabsf(a[0]), len(x01), len(x02), len(x03))) return false;
    float L = fmaxf(abs_sum(x01) + abs_sum(sub(v[1], v[0])), abs_sum(x02) + abs_sum(sub(v[2], v[0])));
    L = fmaxf(L, abs_sum(x03) + abs_sum(sub(v[3], v[0])));
    float c = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) c = fmaxf(c, abs_max(x[k]) + abs_max(v[k]));
    const float line = L * L * (2e-5f + 4e-5f * (c + L));
    const float c1 = a[0] + a[1] / 3.0f, c2 = a[0] + (2.0f * a[1] + a[2]) / 3.0f, c3 = a[0] + a[1] + a[2] + a[3];
    const bool above = a[0] > line && c1 > line && c2 > line && c3 > line;
    const bool below = a[0] < -line && c1 < -line && c2 < -line && c3 < -line;
    return !(above || below);
}

// Distance, normal n (pointing against the relative motion of the face side)
// and barycentric test of a query's four points at time t.
__device__ __forceinline__ float contact_at(bool face, const F3 x[4], const F3 v[4], float t, F3& n, bool& inside) {
    F3 xt[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) xt[k] = add(x[k], scl(t, v[k]));
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    float d;
    if (face) {
        d = face_distance(xt[0], xt[1], xt[2], xt[3], n, w);
        inside = fminf(-w[1], fminf(-w[2], -w[3])) >= -kUpTo3;
    } else {
        d = edge_distance(xt[0], xt[1], xt[2], xt[3], n, w);
        inside = fminf(w[0], fminf(w[1], fminf(-w[2], -w[3]))) >= -kUpTo3;
    }
    const F3 rel = add(add(scl(w[1], v[1]), scl(w[2], v[2])), scl(w[3], v[3]));
    if (dot(n, rel) > 0) n = scl(-1.0f, n);
    return d;
}

// Earliest contact time in [0, 1] of a point-face (face: point q0, face
// q1..q3) or edge-edge (q0q1 against q2q3) query, 1 when none; n is the
// contact normal.  Contact: the four points coplanar at a root of the cubic,
// within 1e-6 of each other's plane / line and inside by the barycentric test.
__device__ float narrow_test(bool face, const F3 x[4], const F3 v[4], F3& n) {
    float a[4];
    F3 x01, x02, x03;
    volume_cubic(x, v, a, x01, x02, x03);
    n = {0.f, 0.f, 0.f};
    if (coplanar(fabsf(a[0]), len(x01), len(x02), len(x03))) return 1.0f;  // coplanar at t = 0
    float t[3];
    const int nr = cubic_roots(a[3], a[2], a[1], a[0], t);
    for (int i = 0; i < nr; ++i) {
        if (t[i] < -kBelow12 || t[i] > 1) continue;
        bool inside;
        const float d = contact_at(face, x, v, t[i], n, inside);
        if (fabsf(d) <= kBelow6 && inside) return t[i];
    }
    return 1.0f;
}

__device__ __forceinline__ void load_query(const uint32_t ids[4], const float4* x, const float4* xt, F3 p[4], F3 v[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        p[k] = f3(x[ids[k]]);
        v[k] = sub(f3(xt[ids[k]]), p[k]);
    }
}

__device__ __forceinline__ unsigned long long time_key(float t, uint32_t tag) {
    const float tk = t > 0.f ? t : 0.f;
    return ((unsigned long long)__float_as_uint(tk) << 32) | tag;
}

// Order-preserving map of floats to signed ints (for atomic min / max).
__device__ __forceinline__ int ord(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float unord(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__device__ __forceinline__ bool overlap(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    return !(ahi.x < blo.x || alo.x > bhi.x || ahi.y < blo.y || alo.y > bhi.y || ahi.z < blo.z || alo.z > bhi.z);
}

// ------------------------------------------------------------ kernels
struct Dev {
    int nv, ntris, nedges;
    const float4* x;
    const float4* xt;
    const uint4* tri;
    const uint4* tri_edges;
    const uint2* edges;
    const int* vcaller;
    const uint4* stri;  // [ntris] the triangles in tree order
    const int* order;   // [ntris] tree position -> triangle
    // swept boxes: level 0 the triangles in tree order, a node of level l the
    // 32^l triangles from 32^l j on; w lanes: the least and the greatest body
    float4* lo;
    float4* hi;
    int top;  // first level from 1 on of at most 32 nodes
    int off[kMaxLevels], cnt[kMaxLevels];
    int2* groups;  // overlapping pairs of level-1 nodes
    int2* pairs;   // candidate triangles
    int group_cap, pair_cap;
    unsigned int* counters;       // [0] pairs found, [1] group pairs found, [2] marked vertices, [3] steps down the tree
    unsigned long long* vf_best;  // [nv]
    unsigned long long* ee_best;  // [nedges]
    unsigned long long* vwin;     // [nv]
    float4* vf_n;                 // [nv] normal of each vertex's earliest face contact
    float4* ee_n;                 // [nedges]
    float* tI;
    float4* nrm;
};

struct Box {
    float4 lo, hi;
};

__device__ __forceinline__ Box empty_box() {
    return {make_float4(FLT_MAX, FLT_MAX, FLT_MAX, __uint_as_float(0xffffffffu)),
            make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, __uint_as_float(0u))};
}

// Least upper box of a warp's boxes (w lanes included), in every lane.
__device__ __forceinline__ Box warp_box(const Box& b) {
    constexpr unsigned kAll = 0xffffffffu;
    Box r;
    r.lo.x = unord(__reduce_min_sync(kAll, ord(b.lo.x)));
    r.lo.y = unord(__reduce_min_sync(kAll, ord(b.lo.y)));
    r.lo.z = unord(__reduce_min_sync(kAll, ord(b.lo.z)));
    r.lo.w = __uint_as_float(__reduce_min_sync(kAll, __float_as_uint(b.lo.w)));
    r.hi.x = unord(__reduce_max_sync(kAll, ord(b.hi.x)));
    r.hi.y = unord(__reduce_max_sync(kAll, ord(b.hi.y)));
    r.hi.z = unord(__reduce_max_sync(kAll, ord(b.hi.z)));
    r.hi.w = __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(b.hi.w)));
    return r;
}

// Everything below a and b is of one body.
__device__ __forceinline__ bool one_body(const Box& a, const Box& b) {
    const uint32_t body = __float_as_uint(a.lo.w);
    return __float_as_uint(a.hi.w) == body && __float_as_uint(b.lo.w) == body && __float_as_uint(b.hi.w) == body;
}

// The boxes of levels 0 to 2 in one pass, a CTA a level-2 node, and the cleared
// results.
__global__ void __launch_bounds__(kBoxThreads) k_boxes(Dev d) {
    __shared__ Box sub_box[32];
    const int p = blockIdx.x * kBoxThreads + threadIdx.x;
    if (p < kCounters) d.counters[p] = 0;
    if (p < d.nv) {
        d.vf_best[p] = kNone;
        d.vwin[p] = kNone;
    }
    if (p < d.nedges) d.ee_best[p] = kNone;
    if (blockIdx.x * kBoxThreads >= d.ntris) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Box b = empty_box();
    if (p < d.ntris) {
        const uint4 tr = d.stri[p];
        const uint32_t id[3] = {tr.x, tr.y, tr.z};
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const float4 q = s ? d.xt[id[k]] : d.x[id[k]];
                b.lo.x = fminf(b.lo.x, q.x);
                b.lo.y = fminf(b.lo.y, q.y);
                b.lo.z = fminf(b.lo.z, q.z);
                b.hi.x = fmaxf(b.hi.x, q.x);
                b.hi.y = fmaxf(b.hi.y, q.y);
                b.hi.z = fmaxf(b.hi.z, q.z);
            }
        b.lo.w = b.hi.w = __uint_as_float(tr.w);
        d.lo[p] = b.lo;
        d.hi[p] = b.hi;
    }
    b = warp_box(b);
    if (lane == 0) {
        sub_box[warp] = b;
        if (p < d.ntris) {
            d.lo[d.off[1] + (p >> 5)] = b.lo;
            d.hi[d.off[1] + (p >> 5)] = b.hi;
        }
    }
    if (d.top < 2) return;
    __syncthreads();
    if (warp > 0) return;
    b = warp_box(sub_box[lane]);
    if (lane == 0) {
        d.lo[d.off[2] + blockIdx.x] = b.lo;
        d.hi[d.off[2] + blockIdx.x] = b.hi;
    }
}

// The boxes of a level from 3 on, a warp a node.
__global__ void __launch_bounds__(kThreads) k_boxes_up(Dev d, int level) {
    pdl_wait();
    pdl_trigger();
    const int j = (blockIdx.x * kThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (j >= d.cnt[level]) return;
    const int c = 32 * j + lane;
    Box b = empty_box();
    if (c < d.cnt[level - 1]) b = {d.lo[d.off[level - 1] + c], d.hi[d.off[level - 1] + c]};
    b = warp_box(b);
    if (lane == 0) {
        d.lo[d.off[level] + j] = b.lo;
        d.hi[d.off[level] + j] = b.hi;
    }
}

// Pairs of groups (g, h >= g) whose boxes overlap and that are not of one body.
// A step down the tree tests 32 boxes, so the chain of loads is a few steps long
// where a binary tree's was some tens, and a poor order of the bodies costs
// little: a million triangles have 1,024 level-2 nodes, 32 steps.
__global__ void __launch_bounds__(kThreads) k_groups(Dev d) {
    __shared__ unsigned int todo[kThreads / 32][kMaxLevels];
    __shared__ int first[kThreads / 32][kMaxLevels];
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = (blockIdx.x * kThreads + threadIdx.x) >> 5;
    if (g >= d.cnt[1]) return;
    const Box own = {d.lo[d.off[1] + g], d.hi[d.off[1] + g]};
    int l = d.top, at = 0;
    for (unsigned int steps = 1;; ++steps) {
        const int c = at + lane;
        bool hit = false;
        // the last group below node c: ((c + 1) 32^(l-1)) - 1
        if (c < d.cnt[l] && ((long long)(c + 1) << (5 * (l - 1))) > g) {
            const Box b = {d.lo[d.off[l] + c], d.hi[d.off[l] + c]};
            hit = !one_body(own, b) && overlap(own.lo, own.hi, b.lo, b.hi);
        }
        unsigned int m = __ballot_sync(0xffffffffu, hit);
        if (l == 1) {
            if (m) {
                unsigned int slot = 0;
                if (lane == 0) slot = atomicAdd(&d.counters[1], (unsigned)__popc(m));
                slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(m & ((1u << lane) - 1));
                if (hit && slot < (unsigned)d.group_cap) d.groups[slot] = make_int2(g, c);
            }
            m = 0;
        }
        // the next node to go into: here, or the nearest level above that has one
        while (m == 0) {
            if (++l > d.top) {
                if (lane == 0) atomicAdd(&d.counters[3], steps);
                return;
            }
            m = todo[warp][l];
            at = first[warp][l];
        }
        const int bit = __ffs(m) - 1;
        __syncwarp();
        if (lane == 0) {
            todo[warp][l] = m & (m - 1);
            first[warp][l] = at;
        }
        __syncwarp();
        at = 32 * (at + bit);
        --l;
    }
}

__device__ __forceinline__ bool share_vertex(uint4 a, uint4 b) {
    return a.x == b.x || a.x == b.y || a.x == b.z || a.y == b.x || a.y == b.y || a.y == b.z || a.z == b.x ||
           a.z == b.y || a.z == b.z;
}

__device__ __forceinline__ float4 shfl4(float4 a, int from) {
    return make_float4(__shfl_sync(0xffffffffu, a.x, from), __shfl_sync(0xffffffffu, a.y, from),
                       __shfl_sync(0xffffffffu, a.z, from), __shfl_sync(0xffffffffu, a.w, from));
}

// Candidate triangles of the overlapping groups, a warp a pair of groups: a lane
// keeps its triangle of the first group, those of the second that reach into the
// first's box go round, and the hits of all 32 x 32 take one atomic.
__global__ void __launch_bounds__(kThreads) k_pairs(Dev d) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warps = gridDim.x * (kThreads / 32);
    const int ngroups = (int)min(d.counters[1], (unsigned)d.group_cap);
    for (int i = (blockIdx.x * kThreads + threadIdx.x) >> 5; i < ngroups; i += warps) {
        const int2 gh = d.groups[i];
        const int p = 32 * gh.x + lane, q = 32 * gh.y + lane;
        Box a = empty_box(), b = empty_box();
        uint4 ta = {}, tb = {};
        if (p < d.ntris) a = {d.lo[p], d.hi[p]}, ta = d.stri[p];
        if (q < d.ntris) b = {d.lo[q], d.hi[q]}, tb = d.stri[q];
        unsigned int m =
            __ballot_sync(0xffffffffu, overlap(d.lo[d.off[1] + gh.x], d.hi[d.off[1] + gh.x], b.lo, b.hi) && q < d.ntris);
        unsigned int hits = 0;
        for (; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            const float4 blo = shfl4(b.lo, k), bhi = shfl4(b.hi, k);
            const bool over = p < d.ntris && (gh.x != gh.y || lane < k) && ta.w != __float_as_uint(blo.w) &&
                              overlap(a.lo, a.hi, blo, bhi);
            if (!__any_sync(0xffffffffu, over)) continue;
            const uint4 t = make_uint4(__shfl_sync(0xffffffffu, tb.x, k), __shfl_sync(0xffffffffu, tb.y, k),
                                       __shfl_sync(0xffffffffu, tb.z, k), 0u);
            if (over && !share_vertex(ta, t)) hits |= 1u << k;
        }
        if (!__any_sync(0xffffffffu, hits != 0)) continue;
        const int mine = __popc(hits);
        int upto = mine;
#pragma unroll
        for (int s = 1; s < 32; s *= 2) {
            const int o = __shfl_up_sync(0xffffffffu, upto, s);
            if (lane >= s) upto += o;
        }
        unsigned int slot = 0;
        if (lane == 31) slot = atomicAdd(&d.counters[0], (unsigned)upto);
        slot = __shfl_sync(0xffffffffu, slot, 31) + (unsigned)(upto - mine);
        const int A = mine ? d.order[p] : 0;
        for (; hits; hits &= hits - 1, ++slot)
            if (slot < (unsigned)d.pair_cap) d.pairs[slot] = make_int2(A, d.order[32 * gh.y + __ffs(hits) - 1]);
    }
}

// Query r < 24 of a candidate pair: 12 a direction, r % 12 < 3 point-face, else
// edge-edge; ids of its four vertices, where its contact goes and its tag.
struct Query {
    uint32_t ids[4];
    unsigned long long* best;
    uint32_t tag;
    bool face;
};
__device__ __forceinline__ Query get_query(const Dev& d, long long g) {
    const int2 pr = d.pairs[g / 24];
    const int r = (int)(g % 24), q = r % 12;
    const int P = r >= 12 ? pr.y : pr.x, Fc = r >= 12 ? pr.x : pr.y;
    Query o;
    o.face = q < 3;
    if (o.face) {
        const uint4 tp = d.tri[P], tf = d.tri[Fc];
        o.ids[0] = q == 0 ? tp.x : q == 1 ? tp.y : tp.z;
        o.ids[1] = tf.x, o.ids[2] = tf.y, o.ids[3] = tf.z;
        o.best = d.vf_best + o.ids[0];
        o.tag = (uint32_t)Fc;
    } else {
        const uint4 ep = d.tri_edges[P], ef = d.tri_edges[Fc];
        const int i = (q - 3) / 3, j = (q - 3) % 3;
        const uint32_t ea = i == 0 ? ep.x : i == 1 ? ep.y : ep.z, eb = j == 0 ? ef.x : j == 1 ? ef.y : ef.z;
        const uint2 a = d.edges[ea], b = d.edges[eb];
        o.ids[0] = a.x, o.ids[1] = a.y, o.ids[2] = b.x, o.ids[3] = b.y;
        o.best = d.ee_best + ea;
        o.tag = eb;
    }
    return o;
}

// A CTA takes up to kBatch queries at a time: those that may touch (may_touch())
// are listed, point-face from the front and edge-edge from the back, and only
// the listed ones go through the cubic's Newton iterations, 32 of a kind a warp.
// With a query a thread a warp waited for its slowest lane's iterations.
constexpr int kBatch = 4 * kThreads;
__global__ void __launch_bounds__(kThreads) k_narrow(Dev d) {
    __shared__ unsigned short list[kBatch];
    __shared__ int found[2];
    pdl_wait();
    pdl_trigger();
    const int t = threadIdx.x;
    const long long total = 24LL * (long long)min(d.counters[0], (unsigned)d.pair_cap);
    // runs of 32 queries, dealt out to the CTAs in turn: contact is local, and so
    // is the work that the sieve leaves
    const int share = (int)((total + 32LL * gridDim.x - 1) / (32LL * gridDim.x));
    for (int run = 0; run < share; run += kBatch / 32) {
        const int batch = 32 * min(share - run, kBatch / 32);
        auto query_at = [&](int u) { return 32 * ((long long)(run + (u >> 5)) * gridDim.x + blockIdx.x) + (u & 31); };
        if (t < 2) found[t] = 0;
        __syncthreads();
        for (int u = t; u < batch; u += kThreads) {
            if (query_at(u) >= total) break;
            const Query q = get_query(d, query_at(u));
            F3 p[4], v[4];
            load_query(q.ids, d.x, d.xt, p, v);
            if (!may_touch(p, v)) continue;
            const int slot = atomicAdd(&found[q.face ? 0 : 1], 1);
            list[q.face ? slot : kBatch - 1 - slot] = (unsigned short)u;
        }
        __syncthreads();
        const int nf = found[0], ne = found[1], warps_f = (nf + 31) & ~31;
        for (int i = t; i < warps_f + ne; i += kThreads) {
            if (i >= nf && i < warps_f) continue;
            const Query q = get_query(d, query_at(list[i < nf ? i : kBatch - 1 - (i - warps_f)]));
            F3 p[4], v[4], n;
            load_query(q.ids, d.x, d.xt, p, v);
            const float tc = narrow_test(q.face, p, v, n);
            if (tc < 1.0f) atomicMin(q.best, time_key(tc, q.tag));
        }
        __syncthreads();
    }
}

// The normal that narrow_test() gave with the contact time in best: its
// evaluation at that time, or the whole query where the key clamped the time.
__device__ __forceinline__ F3 contact_normal(const Dev& d, bool face, const uint32_t ids[4], unsigned long long best) {
    const float t = __uint_as_float((unsigned int)(best >> 32));
    F3 p[4], v[4], n;
    load_query(ids, d.x, d.xt, p, v);
    bool inside;
    if (t > 0.f) contact_at(face, p, v, t, n, inside);
    else narrow_test(face, p, v, n);
    return n;
}

// Winning contact per touched vertex: smallest (time, source) key, the
// source being the caller id of a point-face contact's point or nv + edge.
__global__ void __launch_bounds__(kThreads) k_mark(Dev d) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.nv && d.vf_best[i] != kNone) {
        const unsigned long long best = d.vf_best[i];
        const uint4 tf = d.tri[(uint32_t)(best & 0xffffffffu)];
        const uint32_t ids[4] = {(uint32_t)i, tf.x, tf.y, tf.z};
        const F3 nn = contact_normal(d, true, ids, best);
        d.vf_n[i] = make_float4(nn.x, nn.y, nn.z, 0.f);
        const uint32_t src = d.vcaller ? (uint32_t)d.vcaller[i] : (uint32_t)i;
        const unsigned long long key = (best & 0xffffffff00000000ull) | src;
        atomicMin(&d.vwin[i], key);
        atomicMin(&d.vwin[tf.x], key);
        atomicMin(&d.vwin[tf.y], key);
        atomicMin(&d.vwin[tf.z], key);
    }
    if (i < d.nedges && d.ee_best[i] != kNone) {
        const unsigned long long best = d.ee_best[i];
        const uint2 a = d.edges[i], b = d.edges[(uint32_t)(best & 0xffffffffu)];
        const uint32_t ids[4] = {a.x, a.y, b.x, b.y};
        const F3 nn = contact_normal(d, false, ids, best);
        d.ee_n[i] = make_float4(nn.x, nn.y, nn.z, 0.f);
        const unsigned long long key = (best & 0xffffffff00000000ull) | (uint32_t)(d.nv + i);
        atomicMin(&d.vwin[a.x], key);
        atomicMin(&d.vwin[a.y], key);
    }
}

// tI, and the normals from the winning contacts (each hit vertex has exactly one
// writer; the others' are cleared).
__global__ void __launch_bounds__(kThreads) k_result(Dev d) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool hit = false;
    if (i < d.nv) {
        hit = d.vwin[i] != kNone;
        d.tI[i] = hit ? 0.5f : 1.0f;
        if (!hit) d.nrm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d.vf_best[i] != kNone) {
            const unsigned long long best = d.vf_best[i];
            const uint4 tf = d.tri[(uint32_t)(best & 0xffffffffu)];
            const uint32_t src = d.vcaller ? (uint32_t)d.vcaller[i] : (uint32_t)i;
            const unsigned long long key = (best & 0xffffffff00000000ull) | src;
            const float4 n = d.vf_n[i];
            const float4 m = make_float4(-n.x, -n.y, -n.z, 0.f);
            if (d.vwin[i] == key) d.nrm[i] = n;
            if (d.vwin[tf.x] == key) d.nrm[tf.x] = m;
            if (d.vwin[tf.y] == key) d.nrm[tf.y] = m;
            if (d.vwin[tf.z] == key) d.nrm[tf.z] = m;
        }
    }
    if (i < d.nedges && d.ee_best[i] != kNone) {
        const unsigned long long key = (d.ee_best[i] & 0xffffffff00000000ull) | (uint32_t)(d.nv + i);
        const uint2 a = d.edges[i];
        if (d.vwin[a.x] == key) d.nrm[a.x] = d.ee_n[i];
        if (d.vwin[a.y] == key) d.nrm[a.y] = d.ee_n[i];
    }
    const unsigned int m = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(&d.counters[2], (unsigned)__popc(m));
}

// CCDKernel (collisionUtil.cu:50-70): a vertex with tI < 1 keeps X and gets
// v = -(d . n) n with d = XTilde - X; the others move to XTilde.  Then the
// fixed-body correction of XTilde and v.
// Nothing where a list of the detection was too short: it runs again, and the
// response with it.
__global__ void __launch_bounds__(kThreads) k_respond(Dev det, int nv, const float* tI, const float4* nrm,
                                                     float4* x, const float4* xt, float4* v, SceneArgs sc) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv || det.counters[0] > (unsigned)det.pair_cap || det.counters[1] > (unsigned)det.group_cap) return;
    const float4 p = x[i], q = xt[i];
    float4 vel = v[i];
    if (tI[i] < 1.0f) {
        const F3 n = f3(nrm[i]);
        const F3 dd = sub(f3(q), f3(p));
        const F3 vn = scl(dot(dd, n), n);
        vel = make_float4(-vn.x, -vn.y, -vn.z, 0.f);
    } else {
        x[i] = q;
    }
    if (sc.nfixed > 0 && sc.xt) {
        float3 X = make_float3(q.x, q.y, q.z), V = make_float3(vel.x, vel.y, vel.z);
        collide_fixed(sc, X, V);
        sc.xt[i] = make_float4(X.x, X.y, X.z, 0.f);
        vel = make_float4(V.x, V.y, V.z, 0.f);
    }
    v[i] = vel;
}

}  // namespace

// ------------------------------------------------------------ host side
namespace {
// Bits 0 .. 9 of x spread to every third bit.
uint64_t spread3(uint64_t x) {
    x = (x | x << 16) & 0x030000FF;
    x = (x | x << 8) & 0x0300F00F;
    x = (x | x << 4) & 0x030C30C3;
    return (x | x << 2) & 0x09249249;
}

struct Extent {
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};

    void add(const float* c) {
        for (int k = 0; k < 3; ++k) {
            lo[k] = std::min(lo[k], c[k]);  // NaN: left out
            hi[k] = std::max(hi[k], c[k]);
        }
    }
    // Morton code of c in this box, 10 bits an axis.
    uint64_t code(const float* c) const {
        uint64_t m = 0;
        for (int k = 0; k < 3; ++k) {
            const float ext = hi[k] - lo[k], u = ext > 0.f ? (c[k] - lo[k]) * (1024.f / ext) : 0.f;
            m |= spread3(u > 0.f ? (uint64_t)std::min(u, 1023.f) : 0) << (2 - k);  // NaN: 0
        }
        return m;
    }
    // Volume with every side at least 1/100 of `side`, so that flat ones count.
    double volume(double side) const {
        double v = 1.0;
        for (int k = 0; k < 3; ++k) v *= std::max((double)hi[k] - lo[k], 0.01 * side);
        return v;
    }
};

// Tree order of the triangles at the positions x: body after body along the
// Morton curve of the scene, a body's triangles along that of its own box, which
// stays as good as it is however the body moves.  (In the order of their numbers,
// 10,000 scattered bodies of 2^3 cells took 6.8 ms a detection and 40,000 of one
// cell 49, against 0.35 and 0.63 this way.)
// Where bodies are mixed in space -- their boxes together more than four times the
// scene's -- a body's neighbours on its curve are far apart, and all triangles
// follow one curve: 33,000 triangles of 300 bodies spread over one box take 650 us
// a detection by body and 180 this way, 200,000 of 40 bodies 1,990 and 490.  Only
// for positions that are now: bodies may all have one place when the surface is
// set and be put into theirs later, and then this order is the worst.
void tree_order(const std::vector<uint4>& tri, const float4* x, bool now, std::vector<int>& order) {
    const int ntris = (int)tri.size();
    std::vector<KeyId> key(ntris), tmp;
    std::vector<float> centre(3 * (size_t)ntris);
    Extent scene;
    for (int t = 0; t < ntris; ++t) {
        const float4 p = x[tri[t].x], q = x[tri[t].y], r = x[tri[t].z];
        float* c = &centre[3 * (size_t)t];
        c[0] = p.x + q.x + r.x;
        c[1] = p.y + q.y + r.y;
        c[2] = p.z + q.z + r.z;
        scene.add(c);
        key[t] = {(uint64_t)tri[t].w, t};
    }
    radix_sort(key, tmp);
    double side = 0.0, bodies = 0.0;
    for (int k = 0; k < 3; ++k) side = std::max(side, (double)scene.hi[k] - scene.lo[k]);
    std::vector<int> start;  // first triangle of each body
    std::vector<Extent> box;
    for (int q = 0; q < ntris; ++q) {
        if (q == 0 || key[q].key != key[q - 1].key) {
            start.push_back(q);
            box.emplace_back();
        }
        box.back().add(&centre[3 * (size_t)key[q].id]);
    }
    start.push_back(ntris);
    for (const Extent& b : box) bodies += b.volume(side);
    const bool mixed = now && bodies > 4.0 * scene.volume(side);  // not finite: false
    std::vector<KeyId> along(box.size());  // bodies along the scene's curve
    for (size_t b = 0; b < box.size(); ++b) {
        float mid[3];
        for (int k = 0; k < 3; ++k) mid[k] = 0.5f * box[b].lo[k] + 0.5f * box[b].hi[k];
        along[b] = {scene.code(mid), (int)b};
    }
    radix_sort(along, tmp);
    for (size_t r = 0; r < along.size(); ++r) {
        const int b = along[r].id;
        for (int q = start[b]; q < start[b + 1]; ++q) {
            const float* c = &centre[3 * (size_t)key[q].id];
            key[q].key = mixed ? scene.code(c) : ((uint64_t)r << 30 | box[b].code(c));
        }
    }
    radix_sort(key, tmp);
    order.resize(ntris);
    for (int q = 0; q < ntris; ++q) order[q] = key[q].id;
}
}  // namespace

CcdSurface build_ccd_surface(int nv, int ntris, const uint32_t* tris, const int* tri_body, const int* viperm,
                             const float4* x, bool now) {
    if (nv <= 0 || ntris < 0 || (ntris > 0 && (!tris || !tri_body)))
        throw Error{PDGB_ERR_INVALID_ARGUMENT, "collision surface: bad sizes or null arrays"};
    CcdSurface s;
    s.nv = nv;
    s.ntris = ntris;
    auto iv = [&](uint32_t c) { return viperm ? (uint32_t)viperm[c] : c; };
    // edges by caller ids (smaller, larger), in ascending order: the sides of all
    // triangles sorted, equal ones one edge
    auto side_key = [&](int t, int k) {  // side 0-1, 0-2 or 1-2
        const uint32_t a = tris[3 * (size_t)t + (k == 2)], b = tris[3 * (size_t)t + (k == 0 ? 1 : 2)];
        return (uint64_t)std::min(a, b) << 32 | std::max(a, b);
    };
    std::vector<KeyId> side, tmp;
    side.reserve(3 * (size_t)ntris);
    s.tri.resize(ntris);
    s.tri_edges.resize(ntris);
    for (int t = 0; t < ntris; ++t) {
        uint32_t c[3] = {tris[3 * (size_t)t], tris[3 * (size_t)t + 1], tris[3 * (size_t)t + 2]};
        for (uint32_t v : c)
            if (v >= (uint32_t)nv)
                throw Error{PDGB_ERR_BAD_MESH, "collision triangle " + std::to_string(t) + " references vertex " +
                                                   std::to_string(v) + " >= num_verts"};
        for (int k = 0; k < 3; ++k) side.push_back({side_key(t, k), t});
        std::sort(c, c + 3);
        s.tri[t] = make_uint4(iv(c[0]), iv(c[1]), iv(c[2]), (uint32_t)tri_body[t]);
        s.tri_edges[t].w = 0u;
    }
    radix_sort(side, tmp);
    for (size_t q = 0; q < side.size(); ++q) {
        const uint64_t key = side[q].key;
        if (q == 0 || key != side[q - 1].key)
            s.edges.push_back(make_uint2(iv((uint32_t)(key >> 32)), iv((uint32_t)(key & 0xffffffffu))));
        const uint32_t id = (uint32_t)(s.edges.size() - 1);
        uint4& e = s.tri_edges[side[q].id];
        if (side_key(side[q].id, 0) == key) e.x = id;
        if (side_key(side[q].id, 1) == key) e.y = id;
        if (side_key(side[q].id, 2) == key) e.z = id;
    }
    if (s.edges.size() + (size_t)nv >= 0xffffffffull)
        throw Error{PDGB_ERR_UNSUPPORTED, "collision surface too large"};
    s.nedges = (int)s.edges.size();
    tree_order(s.tri, x, now, s.order);
    return s;
}

struct CcdContext::Buffers {
    DBuf<uint4> tri, stri, tri_edges;
    DBuf<uint2> edges;
    DBuf<int> order;
    DBuf<float4> lo, hi, vf_n, ee_n, nrm;
    DBuf<unsigned int> counters;
    CcdList groups, pairs;
    DBuf<unsigned long long> vf_best, ee_best, vwin;
    DBuf<float> tI;
    int top = 1, off[kMaxLevels] = {}, cnt[kMaxLevels] = {};
    std::vector<uint4> host_tri;  // for the next order
    // work of the first detection after the order was made (< 0: not known yet; 0: it
    // was made for positions that may have changed since), and detections since
    double base = 0.0;
    int age = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    // copy of the counters; page-locking a buffer takes 150 us, the copy to one that
    // is not a few
    unsigned int *counts = nullptr, *pinned = nullptr, pageable[kCounters] = {};
    ~Buffers() {
        if (ev[0]) cudaEventDestroy(ev[0]);
        if (ev[1]) cudaEventDestroy(ev[1]);
        if (pinned) cudaFreeHost(pinned);
    }
};

CcdContext::CcdContext(const CcdSurface& s, const int* vcaller, cudaStream_t stream, bool once)
    : b_(new Buffers), nv_(s.nv), ntris_(s.ntris), nedges_(s.nedges), vcaller_(vcaller), stream_(stream) {
    Buffers& b = *b_;
    b.tri.upload(s.tri, stream);
    b.tri_edges.upload(s.tri_edges, stream);
    b.edges.upload(s.edges, stream);
    if (!once) b.host_tri = s.tri;
    upload_order(s.tri, s.order);
    size_t nodes = 0;
    for (int l = 0; l < kMaxLevels; ++l) {
        b.cnt[l] = l == 0 ? ntris_ : (b.cnt[l - 1] + 31) / 32;
        b.off[l] = (int)nodes;
        nodes += (size_t)b.cnt[l];
        if (nodes > 0x7fffffff) throw Error{PDGB_ERR_UNSUPPORTED, "collision surface too large"};
    }
    while (b.cnt[b.top] > 32) ++b.top;
    b.lo.alloc(std::max<size_t>(nodes, 1));
    b.hi.alloc(std::max<size_t>(nodes, 1));
    b.counters.alloc(kCounters);
    if (!once) PDGB_CUDA_TRY(cudaMallocHost(&b.pinned, kCounters * sizeof(unsigned int)));
    b.counts = b.pinned ? b.pinned : b.pageable;
    const size_t n = (size_t)std::max(ntris_, 1);
    b.groups.least = std::max(16 * b.cnt[1], 256);
    b.groups.ensure();
    b.pairs.least = (int)std::min<size_t>(std::max<size_t>(16 * n, 4096), kMostPairs);
    b.pairs.ensure();
    b.vf_best.alloc(nv_);
    b.vwin.alloc(nv_);
    b.vf_n.alloc(nv_);
    b.ee_best.alloc(std::max(nedges_, 1));
    b.ee_n.alloc(std::max(nedges_, 1));
    b.tI.alloc(nv_);
    b.nrm.alloc(nv_);
    PDGB_CUDA_TRY(cudaEventCreate(&b.ev[0]));
    PDGB_CUDA_TRY(cudaEventCreate(&b.ev[1]));
    // no contact until the first detection
    std::vector<float> ones(nv_, 1.0f);
    PDGB_CUDA_TRY(cudaMemcpyAsync(b.tI.p, ones.data(), nv_ * sizeof(float), cudaMemcpyHostToDevice, stream));
    PDGB_CUDA_TRY(cudaMemsetAsync(b.nrm.p, 0, nv_ * sizeof(float4), stream));
    PDGB_CUDA_TRY(cudaStreamSynchronize(stream));
}

CcdContext::~CcdContext() = default;

void CcdContext::upload_order(const std::vector<uint4>& tri, const std::vector<int>& order) {
    std::vector<uint4> sorted(ntris_);
    for (int q = 0; q < ntris_; ++q) sorted[q] = tri[order[q]];
    b_->stri.upload(sorted, stream_);
    b_->order.upload(order, stream_);
    PDGB_CUDA_TRY(cudaStreamSynchronize(stream_));
}

// The order is as good as the positions that it was made at.  A detection counts
// what it costs: the steps down the tree and the pairs of groups, some 5 to 60 a
// group where bodies touch or fly about.  Where it is more, and this is the first
// detection, or some steps later one that takes four times what it took when the
// order was made, or a thousand steps later, the triangles are ordered anew where
// they are now.  2,000 bodies of 5^3 cells that shared one place when the surface
// was set and were then put into theirs take 26 ms for the first step (20 of them
// this, on the host) and 0.75 from the second on; 3.0 in a tree built for each.
constexpr double kPoorWork = 64.0;
constexpr int kOrderAge = 1000, kOrderRest = 16;

void CcdContext::keep_order(const float4* x) {
    Buffers& b = *b_;
    if (b.host_tri.empty() || b.top < 2) return;  // up to 32 groups are one step
    const double work = (double)b.counts[3] + 4.0 * b.counts[1];
    if (b.base < 0.0) b.base = work;  // the first in this order
    ++b.age;
    if (work < kPoorWork * b.cnt[1]) return;
    // not every other step where two kinds of steps take turns
    const bool grown = work >= 4.0 * b.base && (b.base == 0.0 || b.age >= kOrderRest);
    if (!grown && b.age < kOrderAge) return;
    try {
        std::vector<float4> h(nv_);
        PDGB_CUDA_TRY(cudaMemcpyAsync(h.data(), x, (size_t)nv_ * sizeof(float4), cudaMemcpyDeviceToHost, stream_));
        PDGB_CUDA_TRY(cudaStreamSynchronize(stream_));
        std::vector<int> order;
        tree_order(b.host_tri, h.data(), true, order);
        upload_order(b.host_tri, order);
    } catch (const std::bad_alloc&) {  // the present order is as right
    }
    b.base = -1.0;
    b.age = 0;
}

const float* CcdContext::tI() const { return b_->tI.p; }
const float4* CcdContext::normals() const { return b_->nrm.p; }

void CcdContext::detect(const float4* x, const float4* xt, const CcdResponse* response) {
    Buffers& b = *b_;
    cudaStream_t s = stream_;
    PDGB_CUDA_TRY(cudaEventRecord(b.ev[0], s));
    Dev d{};
    d.nv = nv_;
    d.ntris = ntris_;
    d.nedges = nedges_;
    d.x = x;
    d.xt = xt;
    d.tri = b.tri.p;
    d.tri_edges = b.tri_edges.p;
    d.edges = b.edges.p;
    d.vcaller = vcaller_;
    d.stri = b.stri.p;
    d.order = b.order.p;
    d.lo = b.lo.p;
    d.hi = b.hi.p;
    d.top = b.top;
    std::copy(b.off, b.off + kMaxLevels, d.off);
    std::copy(b.cnt, b.cnt + kMaxLevels, d.cnt);
    d.counters = b.counters.p;
    d.vf_best = b.vf_best.p;
    d.ee_best = b.ee_best.p;
    d.vwin = b.vwin.p;
    d.vf_n = b.vf_n.p;
    d.ee_n = b.ee_n.p;
    d.tI = b.tI.p;
    d.nrm = b.nrm.p;
    const int most = std::max({nv_, nedges_, ntris_, kCounters});
    const int outs = blocks_for(std::max(nv_, nedges_));
    // The lists grow to the counts found and the detection runs again: the count
    // of pairs is whole once the list of groups is.
    for (int attempt = 0;; ++attempt) {
        b.groups.ensure();
        b.pairs.ensure();
        d.groups = b.groups.items.p;
        d.pairs = b.pairs.items.p;
        d.group_cap = b.groups.cap;
        d.pair_cap = b.pairs.cap;
        k_boxes<<<(int)(((long long)most + kBoxThreads - 1) / kBoxThreads), kBoxThreads, 0, s>>>(d);
        if (ntris_ >= 2) {
            for (int l = 3; l <= b.top; ++l) launch_pdl(k_boxes_up, blocks_for(32LL * b.cnt[l]), kThreads, 0, s, d, l);
            launch_pdl(k_groups, blocks_for(32LL * b.cnt[1]), kThreads, 0, s, d);
            launch_pdl(k_pairs, (int)std::min<long long>(blocks_for(32LL * b.groups.cap), kListCtas), kThreads, 0, s, d);
            launch_pdl(k_narrow, (int)std::min<long long>(blocks_for(24LL * b.pairs.cap), kListCtas), kThreads, 0, s, d);
        }
        launch_pdl(k_mark, outs, kThreads, 0, s, d);
        launch_pdl(k_result, outs, kThreads, 0, s, d);
        PDGB_CUDA_TRY(cudaGetLastError());
        PDGB_CUDA_TRY(cudaEventRecord(b.ev[1], s));
        if (response)
            launch_pdl(k_respond, blocks_for(nv_), kThreads, 0, s, d, nv_, b.tI.p, b.nrm.p, response->x, xt, response->v,
                       response->sc);
        PDGB_CUDA_TRY(cudaMemcpyAsync(b.counts, b.counters.p, kCounters * sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
        PDGB_CUDA_TRY(cudaStreamSynchronize(s));
        const bool groups = b.counts[1] > (unsigned)b.groups.cap, pairs = b.counts[0] > (unsigned)b.pairs.cap;
        if (!groups && !pairs) break;
        if (attempt > 1 || std::max(b.counts[0], b.counts[1]) > kMostPairs)
            throw Error{PDGB_ERR_OUT_OF_MEMORY, "too many collision candidates"};
        if (groups) {
            b.groups.grow((long long)b.counts[1] + b.counts[1] / 4);
        } else {
            b.pairs.grow((long long)b.counts[0] + b.counts[0] / 4);
            stats_.regrows++;
        }
    }
    float ms = 0.f;
    PDGB_CUDA_TRY(cudaEventElapsedTime(&ms, b.ev[0], b.ev[1]));
    stats_.pairs = b.counts[0];
    stats_.marked = (int)b.counts[2];
    stats_.ms = ms;
    if (ntris_ >= 2) keep_order(x);
}

}  // namespace pdgb
