// Device building blocks of the ptnee wavefront: vector helpers, the Philox
// path stream, the reference-exact ray/box and ray/triangle tests and the
// BVH traversals. Included by the .cu files of libnuray_gpu.so only.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

#include "nr_types.h"

namespace nr {

// ------------------------------------------------------------------ vectors
struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 mk(float s) { return {s, s, s}; }
__device__ __forceinline__ f3 xyz(float4 v) { return {v.x, v.y, v.z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ f3 operator*(f3 a, f3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator*(float s, f3 a) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator/(f3 a, float s) { return {a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float norm2(f3 a) { return dot(a, a); }
__device__ __forceinline__ float norm(f3 a) { return sqrtf(norm2(a)); }
// vec3::normalized divides by |a| + 1e-8 (src/math/vec3.cpp:70-73)
__device__ __forceinline__ f3 normalized(f3 a) { return a / (norm(a) + 1e-8f); }
// std::max / std::min semantics (first argument kept unless strictly beaten)
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }

// Rounded-to-nearest float ops that the compiler may not fuse; used where the
// reference's FP32 results have to be reproduced bit for bit.
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ f3 rsub3(f3 a, f3 b) { return {rsub(a.x, b.x), rsub(a.y, b.y), rsub(a.z, b.z)}; }
__device__ __forceinline__ float rdot(f3 a, f3 b) { return radd(radd(rmul(a.x, b.x), rmul(a.y, b.y)), rmul(a.z, b.z)); }
__device__ __forceinline__ f3 rcross(f3 a, f3 b) {
    return {rsub(rmul(a.y, b.z), rmul(a.z, b.y)), rsub(rmul(a.z, b.x), rmul(a.x, b.z)),
            rsub(rmul(a.x, b.y), rmul(a.y, b.x))};
}

// Correctly rounded a / b given rb = RN(1/b): one residual correction of
// the product a * rb (Markstein). Exact for finite, non-denormal results.
__device__ __forceinline__ float qdiv(float a, float b, float rb) {
    float q0 = __fmul_rn(a, rb);
    float r = __fmaf_rn(-q0, b, a);
    return __fmaf_rn(r, rb, q0);
}

// RN_float(x + 1e-6) where 1e-6 is the double literal of the reference's
// `s1.dot(e1) + 1e-6` (src/scene/triangle.cpp:31): a float TwoSum with the
// split constant hi + lo. Differs from the double evaluation only when the
// exact sum lies within 2^-48 of a float rounding boundary.
__device__ __forceinline__ float add_1e6(float x) {
    const float hi = 9.99999997475242708e-07f;
    const float lo = (float)(1e-6 - (double)9.99999997475242708e-07f);
    float s = __fadd_rn(x, hi);
    float bb = __fsub_rn(s, x);
    float e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(hi, bb));
    return __fadd_rn(s, __fadd_rn(e, lo));
}

// ------------------------------------------------------------------ Philox
// Philox4x32-10 (Salmon et al., SC'11). Path stream: draw n of path
// (pixel, sample) is lane n%4 of philox(ctr = (pixel, sample, n/4, tag),
// key = seed); uniform = (x >> 8) * 2^-24.
#define NR_STREAM_TAG 0x6e755279u
__device__ __forceinline__ uint4 philox10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

struct Stream {
    uint2 key;
    uint32_t pixel, sample, n;
    uint4 buf;
    __device__ __forceinline__ void init(uint32_t seed_lo, uint32_t seed_hi, uint32_t px, uint32_t smp, uint32_t first) {
        key = make_uint2(seed_lo, seed_hi);
        pixel = px; sample = smp; n = first;
        buf = philox10(make_uint4(pixel, sample, n >> 2, NR_STREAM_TAG), key);
    }
    __device__ __forceinline__ float next() {
        if ((n & 3u) == 0u && n != 0u) buf = philox10(make_uint4(pixel, sample, n >> 2, NR_STREAM_TAG), key);
        uint32_t lane = n & 3u;
        uint32_t x = lane == 0 ? buf.x : (lane == 1 ? buf.y : (lane == 2 ? buf.z : buf.w));
        ++n;
        return (float)(x >> 8) * (1.0f / 16777216.0f);
    }
};

// ------------------------------------------------------------------ intersection
// Ray prepared for the exact slab test: denominators d + 1e-9f and their
// correctly rounded reciprocals (src/hierarchy/bvhnode.cpp:41).
struct SlabRay {
    float ox, oy, oz;
    float dx, dy, dz;     // d + 1e-9f
    float rx, ry, rz;     // RN(1 / (d + 1e-9f))
    float cx, cy, cz;     // RN(-o * r), for the one-FMA approximate quotient; NaN where r is infinite
    float abs_err;        // bound on |fma(b, r, c) - (b - o) r| from rounding c
};
__device__ __forceinline__ SlabRay make_slab_ray(f3 o, f3 d) {
    SlabRay r;
    r.ox = o.x; r.oy = o.y; r.oz = o.z;
    r.dx = __fadd_rn(d.x, 1e-9f); r.dy = __fadd_rn(d.y, 1e-9f); r.dz = __fadd_rn(d.z, 1e-9f);
    r.rx = __frcp_rn(r.dx); r.ry = __frcp_rn(r.dy); r.rz = __frcp_rn(r.dz);
    // A component of exactly -1e-9f leaves a denominator of 0 and an infinite
    // r. qdiv's quotients are then NaN, which smax and smin pass over: the exact
    // test leaves that axis out. With -o r one plane of a box that holds the
    // origin would be infinite and the other NaN, and a minimum that drops the
    // NaN puts both on one side; r - r is 0 for every finite r and NaN for this
    // one, so the quotients below are NaN and their tests leave the axis out too.
    r.cx = __fmaf_rn(-o.x, r.rx, __fsub_rn(r.rx, r.rx));
    r.cy = __fmaf_rn(-o.y, r.ry, __fsub_rn(r.ry, r.ry));
    r.cz = __fmaf_rn(-o.z, r.rz, __fsub_rn(r.rz, r.rz));
    // |c| * 2^-24 (rounding of c) with headroom: 2^-22
    r.abs_err = 2.4e-7f * fmaxf(fabsf(r.cx), fmaxf(fabsf(r.cy), fabsf(r.cz)));
    return r;
}

// BVHNode::intersect (src/hierarchy/bvhnode.cpp:35-48) with the same
// rounding: t = (bound - o) / (d + 1e-9f), swap, std::max / std::min.
// Returns the entry distance in *tin when accepted.
__device__ __forceinline__ bool slab_axis(float lo, float hi, float o, float d, float rd, float& tin, float& tout) {
    float t1 = qdiv(__fsub_rn(lo, o), d, rd);
    float t2 = qdiv(__fsub_rn(hi, o), d, rd);
    if (t1 > t2) { float s = t1; t1 = t2; t2 = s; }
    tin = smax(tin, t1);
    tout = smin(tout, t2);
    return true;
}
__device__ __forceinline__ bool box_test(const SlabRay& r, float lx, float hx, float ly, float hy, float lz, float hz,
                                         float& t_entry) {
    float tin = -1e18f, tout = 1e18f;
    slab_axis(lx, hx, r.ox, r.dx, r.rx, tin, tout);
    slab_axis(ly, hy, r.oy, r.dy, r.ry, tin, tout);
    slab_axis(lz, hz, r.oz, r.dz, r.rz, tin, tout);
    t_entry = tin;
    return tin <= tout && tout >= 0.0f;
}

// The same decision from approximate quotients (b - o) * RN(1/d): each is
// within 2^-22.4 of the exact quotient, and the sign is exact, so the result
// can only differ from the exact test when the entry and exit distances lie
// within that error of each other; those cases are recomputed exactly.
__device__ __forceinline__ bool box_test_fast(const SlabRay& r, float lx, float hx, float ly, float hy, float lz, float hz,
                                              float& t_entry) {
    // one FMA per bound: fma(b, r, -o r) is within 2^-22.4 |q| + abs_err of
    // the exact quotient q = (b - o) / d
    float x1 = __fmaf_rn(lx, r.rx, r.cx), x2 = __fmaf_rn(hx, r.rx, r.cx);
    float y1 = __fmaf_rn(ly, r.ry, r.cy), y2 = __fmaf_rn(hy, r.ry, r.cy);
    float z1 = __fmaf_rn(lz, r.rz, r.cz), z2 = __fmaf_rn(hz, r.rz, r.cz);
    float tin = fmaxf(fmaxf(fminf(x1, x2), fminf(y1, y2)), fmaxf(fminf(z1, z2), -1e18f));
    float tout = fminf(fminf(fmaxf(x1, x2), fmaxf(y1, y2)), fminf(fmaxf(z1, z2), 1e18f));
    float margin = 1e-6f * fmaxf(fabsf(tin), fabsf(tout)) + r.abs_err;
    if (tout < -margin) return false;
    if (tin + margin < tout && tout > margin) { t_entry = tin; return true; }
    if (tin > tout + margin) return false;
    return box_test(r, lx, hx, ly, hy, lz, hz, t_entry);
}

// Box test of the binary walks: FAST the one-FMA test with its error margin
// and exact fallback, else the reference's arithmetic throughout (the same
// answers).
template <bool FAST>
__device__ __forceinline__ bool box_test_mode(const SlabRay& r, float lx, float hx, float ly, float hy, float lz, float hz,
                                              float& t_entry) {
    return FAST ? box_test_fast(r, lx, hx, ly, hy, lz, hz, t_entry) : box_test(r, lx, hx, ly, hy, lz, hz, t_entry);
}

// Triangle::intersection (src/scene/triangle.cpp:27-33) followed by the leaf
// acceptance test of BVHNode::getIntersection (src/hierarchy/bvhnode.cpp:55-63):
// t < limit && t > 0 && b1 >= 0 && b2 >= 0 && b1 + b2 <= 1.
__device__ __forceinline__ bool tri_test(f3 o, f3 d, float4 g0, float4 g1, float4 g2, float limit, float& t, float& b1,
                                         float& b2) {
    f3 p0 = xyz(g0), e1 = xyz(g1), e2 = xyz(g2);
    f3 s = rsub3(o, p0);
    f3 s1 = rcross(d, e2);
    f3 s2 = rcross(s, e1);
    float tt = rdot(s2, e2);
    float q = add_1e6(rdot(s1, e1));
    // t = tt / q > 0 needs equal signs and tt != 0; anything else is rejected.
    if (tt == 0.0f || ((__float_as_uint(tt) ^ __float_as_uint(q)) & 0x80000000u)) return false;
    float rq = __frcp_rn(q);
    t = qdiv(tt, q, rq);
    if (!(t < limit && t > 0.0f)) return false;
    b1 = qdiv(rdot(s1, s), q, rq);
    b2 = qdiv(rdot(s2, d), q, rq);
    return b1 >= 0.0f && b2 >= 0.0f && __fadd_rn(b1, b2) <= 1.0f;
}

// tri_test with an approximate reciprocal of q: the decision is taken from
// quotients within 2^-21 of the exact ones when every comparison clears that
// margin, and recomputed with the exact division otherwise, so the accepted
// set and the returned t, b1, b2 equal tri_test's.
__device__ __forceinline__ bool tri_test_fast(f3 o, f3 d, float4 g0, float4 g1, float4 g2, float limit, float& t,
                                              float& b1, float& b2) {
    f3 p0 = xyz(g0), e1 = xyz(g1), e2 = xyz(g2);
    const float e = 1e-6f, tiny = 1e-30f;
    // The rejections in the order of what they need, so a miss on the first
    // barycentric skips the second cross product: the same rejections as the
    // exact test's, all of them checked before a hit is kept (1M-triangle
    // frame: 706.1 -> 717.1 Mpaths/s against computing all before rejecting).
    f3 s1 = rcross(d, e2);
    float q = add_1e6(rdot(s1, e1));
    f3 s = rsub3(o, p0);
    float u = rdot(s1, s);
    // quotients from an approximate reciprocal (2 ulp): within 2^-21 of the exact ones
    float rq = __fdividef(1.0f, q);
    float ua = u * rq;
    // with va >= -tiny, ua > 1 + 2e already puts the rounded ua + va above 1 + 2e
    if (ua < -tiny || ua > 1.0f + 2.0f * e) return false;
    f3 s2 = rcross(s, e1);
    float v = rdot(s2, d);
    float va = v * rq;
    if (va < -tiny || ua + va > 1.0f + 2.0f * e) return false;
    float tt = rdot(s2, e2);
    // t = tt / q > 0 needs equal signs and tt != 0 (exact)
    if (tt == 0.0f || ((__float_as_uint(tt) ^ __float_as_uint(q)) & 0x80000000u)) return false;
    float ta = tt * rq;
    if (ta > limit * (1.0f + e)) return false;
    float rqe = __frcp_rn(q);
    if (ta < limit * (1.0f - e) && ta > tiny && ua > tiny && va > tiny && ua + va < 1.0f - 2.0f * e) {
        t = qdiv(tt, q, rqe);
        b1 = qdiv(u, q, rqe);
        b2 = qdiv(v, q, rqe);
        return true;
    }
    // close to an edge, the far limit or zero: decide with the exact quotients
    t = qdiv(tt, q, rqe);
    if (!(t < limit && t > 0.0f)) return false;
    b1 = qdiv(u, q, rqe);
    b2 = qdiv(v, q, rqe);
    return b1 >= 0.0f && b2 >= 0.0f && __fadd_rn(b1, b2) <= 1.0f;
}

// Pruning: a subtree whose entry distance exceeds the best hit so far (or a
// shadow ray's limit) times S.prune_k is skipped; the reference prunes
// nothing (src/hierarchy/bvh.cpp:116-117). The default factor is
// 1 + NR_PRUNE_MARGIN. The reference's biased determinant (q + 1e-6,
// src/scene/triangle.cpp:31) reports t' = t q / (q + 1e-6) and accepts the
// triangle scaled about p0 by (q + 1e-6) / q, so a triangle crossed at a
// grazing angle (0 < q < 1e-6 / margin, or |q| < 1e-6) can report a t
// below its box's entry distance, even below the best hit of another
// subtree; no bound from the boxes excludes it. Such rays need the plane
// of a triangle to hold the ray to about 1e-6 of its length; prune=0
// (S.prune_k = infinity) visits every node whose box the ray enters, as
// the reference does, and returns the reference's hits for them too.
// LightSampler::sampleLight (src/sampler/lightsampler.cpp:56): the first
// emitter whose CDF entry is >= r (lower_bound), or the last one. The guide
// table narrows the search to the emitters between the lower bounds of
// floor(r K) / K and (floor(r K) + 1) / K, which enclose the answer.
__device__ __forceinline__ int pick_light(const DeviceScene& S, float r) {
    const int k = S.light_guide_k;
    int b = (int)(r * (float)k);
    b = b < 0 ? 0 : (b > k - 1 ? k - 1 : b);
    int lo = __ldg(&S.light_guide[b]), hi = __ldg(&S.light_guide[b + 1]);
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&S.light_cdf[mid]) < r) lo = mid + 1; else hi = mid;
    }
    return lo < S.num_lights ? lo : S.num_lights - 1;
}

#define NR_STACK NR_STACK_LIMIT

// Closest hit with the reference's exhaustive semantics (BVH::_traversal,
// src/hierarchy/bvh.cpp:99-127): the minimum t over reachable triangles;
// equal t resolved towards the later leaf in depth-first order (the
// reference keeps the right subtree unless the left is strictly nearer) and,
// within a leaf, towards the earlier triangle. Visits children near-first
// and prunes with the margin above. Returns the flattened triangle index or
// -1; err is set on a stack overflow.
template <bool FAST = true>
__device__ __forceinline__ int closest_hit(const DeviceScene& S, f3 o, f3 d, float& best_t, float& best_b1,
                                           float& best_b2, uint32_t* err, uint32_t* nodes_visited = nullptr,
                                           uint32_t* tris_tested = nullptr) {
    best_t = 1e18f; best_b1 = 0.f; best_b2 = 0.f;
    int best = -1, best_leaf = -1;
    if (S.root_ref == INT32_MIN) return -1;
    SlabRay R = make_slab_ray(o, d);
    float te;
    if (!box_test(R, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return -1;
    // (subtree reference, entry distance) pairs: one 8-byte local access per push / pop
    int2 stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    uint32_t nv = 0, nt = 0;
    // every node is entered at most once per ray; the cap only guards against
    // a corrupted node array
    int budget = 2 * S.num_nodes + 8;
    while (true) {
        if (--budget < 0) { atomicOr(err, 2u); break; }
        if (ref >= 0) {
            const GpuNode& N = S.nodes[ref];
            float4 a = __ldg(&N.a), b = __ldg(&N.b), c = __ldg(&N.c);
            int4 k = __ldg(&N.d);
            ++nv;
            float t0, t1;
            bool h0 = FAST ? box_test_fast(R, a.x, a.y, a.z, a.w, c.x, c.y, t0) : box_test(R, a.x, a.y, a.z, a.w, c.x, c.y, t0);
            bool h1 = FAST ? box_test_fast(R, b.x, b.y, b.z, b.w, c.z, c.w, t1) : box_test(R, b.x, b.y, b.z, b.w, c.z, c.w, t1);
            float lim = best_t * S.prune_k;
            h0 = h0 && t0 <= lim;
            h1 = h1 && t1 <= lim;
            if (h0 && h1) {
                int nr = k.x, fr = k.y;
                float ft = t1;
                if (t1 < t0) { nr = k.y; fr = k.x; ft = t0; }
                if (sp >= NR_STACK) { atomicOr(err, 1u); break; }
                stack[sp] = make_int2(fr, __float_as_int(ft)); ++sp;
                ref = nr;
                continue;
            }
            if (h0) { ref = k.x; continue; }
            if (h1) { ref = k.y; continue; }
        } else {
            int first = leaf_first(ref), cnt = leaf_count(ref);
            float lt = 1e18f;
            int li = -1;
            for (int i = 0; i < cnt; ++i) {
                int ti = first + i;
                float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
                ++nt;
                float t, u, v;
                if (FAST ? tri_test_fast(o, d, g0, g1, g2, lt, t, u, v) : tri_test(o, d, g0, g1, g2, lt, t, u, v)) {
                    lt = t; li = ti;
                }
            }
            if (li >= 0 && (lt < best_t || (lt == best_t && first > best_leaf))) {
                best_t = lt; best = li; best_leaf = first;
            }
        }
        // pop the next subtree that can still hold a hit
        bool found = false;
        while (sp > 0) {
            --sp;
            const int2 e = stack[sp];
            if (__int_as_float(e.y) <= best_t * S.prune_k) { ref = e.x; found = true; break; }
        }
        if (!found) break;
    }
    if (nodes_visited) *nodes_visited += nv;
    if (tris_tested) *tris_tested += nt;
    if (best >= 0) {
        // barycentrics of the winner, recomputed rather than carried through
        // the loop (fewer live registers): both tests return the correctly
        // rounded quotients, so these equal the values found in the leaf
        float4 g0 = __ldg(&S.tri_geo[3 * best]), g1 = __ldg(&S.tri_geo[3 * best + 1]), g2 = __ldg(&S.tri_geo[3 * best + 2]);
        float t;
        tri_test(o, d, g0, g1, g2, 3.0e38f, t, best_b1, best_b2);
    }
    return best;
}

// Refs: inner nodes >= 0, leaves < 0; NR_TRAV_END (no node) ends a walk.
#define NR_TRAV_END 0x7fffffff

// The walk of trav=0, with the reference's boxes and arithmetic throughout:
// while-while with postponed leaves (Aila and Laine, "Understanding the
// efficiency of ray traversal on GPUs", HPG 2009). A lane that reaches a leaf
// keeps it aside and goes on through inner nodes until every active lane of
// its warp holds a leaf; then the warp tests leaves together. Same hits as
// closest_hit: the winner is the minimum t, ties to the larger leaf start and
// then the earlier triangle of the leaf, whatever the visiting order, and a
// subtree is only skipped when its entry distance exceeds the pruning limit
// of the best hit so far, which never undercuts the final one.
// No step budget and no stack-full test: the host accepts only trees in
// which every inner node has at most one parent, of a smaller index, and
// whose depth leaves the stack room (upload_scene and finish_scene), so a
// walk visits each node at most once and its stack holds at most one entry
// per level.
__device__ __forceinline__ int closest_hit_ww(const DeviceScene& S, f3 o, f3 d, float& best_t, float& best_b1,
                                              float& best_b2, uint32_t* nodes_visited = nullptr,
                                              uint32_t* tris_tested = nullptr) {
    best_t = 1e18f; best_b1 = 0.f; best_b2 = 0.f;
    int best = -1, best_leaf = -1;
    if (S.root_ref == INT32_MIN) return -1;
    SlabRay R = make_slab_ray(o, d);
    float te;
    if (!box_test(R, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return -1;
    int2 stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    int leaf = 0;  // postponed leaf (< 0), or none (>= 0)
    if (ref < 0) { leaf = ref; ref = NR_TRAV_END; }  // the whole scene is one leaf
    uint32_t nv = 0, nt = 0;
    // the next stacked subtree that can still hold a hit, or NR_TRAV_END
    auto pop = [&]() {
        while (sp > 0) {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) <= best_t * S.prune_k) return e.x;
        }
        return (int)NR_TRAV_END;
    };
    while (ref != NR_TRAV_END || leaf < 0) {
        while ((unsigned)ref < (unsigned)NR_TRAV_END) {
            const GpuNode& N = S.nodes[ref];
            float4 a = __ldg(&N.a), b = __ldg(&N.b), c = __ldg(&N.c);
            int4 k = __ldg(&N.d);
            ++nv;
            float t0, t1;
            bool h0 = box_test(R, a.x, a.y, a.z, a.w, c.x, c.y, t0);
            bool h1 = box_test(R, b.x, b.y, b.z, b.w, c.z, c.w, t1);
            const float lim = best_t * S.prune_k;
            h0 = h0 && t0 <= lim;
            h1 = h1 && t1 <= lim;
            if (h0 && h1) {
                int nr = k.x, fr = k.y;
                float ft = t1;
                if (t1 < t0) { nr = k.y; fr = k.x; ft = t0; }
                stack[sp++] = make_int2(fr, __float_as_int(ft));
                ref = nr;
            } else if (h0) {
                ref = k.x;
            } else if (h1) {
                ref = k.y;
            } else {
                ref = pop();
            }
            if (ref < 0 && leaf >= 0) {  // first leaf: keep it aside, go on
                leaf = ref;
                ref = pop();
            }
            if (!__any_sync(__activemask(), leaf >= 0)) break;
        }
        while (leaf < 0) {
            int first = leaf_first(leaf), cnt = leaf_count(leaf);
            float lt = 1e18f;
            int li = -1;
            for (int i = 0; i < cnt; ++i) {
                int ti = first + i;
                float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
                ++nt;
                float t, u, v;
                const float cap = fminf(lt, __uint_as_float(__float_as_uint(best_t) + 1u));
                if (tri_test(o, d, g0, g1, g2, cap, t, u, v)) { lt = t; li = ti; }
            }
            if (li >= 0 && (lt < best_t || (lt == best_t && first > best_leaf))) {
                best_t = lt; best = li; best_leaf = first;
            }
            // a second leaf reached while this one waited goes next
            leaf = ref;
            if (ref < 0) ref = pop();
        }
    }
    if (nodes_visited) *nodes_visited += nv;
    if (tris_tested) *tris_tested += nt;
    if (best >= 0) {
        float4 g0 = __ldg(&S.tri_geo[3 * best]), g1 = __ldg(&S.tri_geo[3 * best + 1]), g2 = __ldg(&S.tri_geo[3 * best + 2]);
        float t;
        tri_test(o, d, g0, g1, g2, 3.0e38f, t, best_b1, best_b2);
    }
    return best;
}

// Shadow query on the reference's boxes: true when some reachable triangle
// has a reference hit with t <= tmax (the complement of `t + 2e-3 >
// |light_vec|` of src/renderer/rendererptls.cpp:71 for the closest hit).
// While-while: a lane's inner-node loop ends at its first leaf. FAST: the
// tests with the exact fallback; both give the same answer.
template <bool FAST>
__device__ __forceinline__ bool any_hit_ww(const DeviceScene& S, f3 o, f3 d, float tmax, uint32_t* err,
                                           uint32_t* nodes_visited = nullptr, uint32_t* tris_tested = nullptr) {
    if (S.root_ref == INT32_MIN) return false;
    SlabRay R = make_slab_ray(o, d);
    float te;
    if (!box_test(R, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return false;
    const float lim = tmax * S.prune_k;
    int stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    const float limit = fminf(1e18f, __uint_as_float(__float_as_uint(tmax) + 1u));  // accepts t <= tmax
    int budget = 2 * S.num_nodes + 8;
    while (true) {
        while (ref >= 0) {
            if (--budget < 0) { atomicOr(err, 2u); return false; }
            const GpuNode& N = S.nodes[ref];
            float4 a = __ldg(&N.a), b = __ldg(&N.b), c = __ldg(&N.c);
            int4 k = __ldg(&N.d);
            if (nodes_visited) ++*nodes_visited;
            float t0, t1;
            const bool h0 = box_test_mode<FAST>(R, a.x, a.y, a.z, a.w, c.x, c.y, t0) && t0 <= lim;
            const bool h1 = box_test_mode<FAST>(R, b.x, b.y, b.z, b.w, c.z, c.w, t1) && t1 <= lim;
            if (h0 && h1) {
                int nr = k.x, fr = k.y;
                // far child first: the near one holds the surface the shadow
                // ray leaves and its neighbours, which seldom occlude it
                if (t1 > t0) { nr = k.y; fr = k.x; }
                if (sp >= NR_STACK) { atomicOr(err, 1u); return false; }
                stack[sp++] = fr;
                ref = nr;
            } else if (h0) {
                ref = k.x;
            } else if (h1) {
                ref = k.y;
            } else {
                if (sp == 0) return false;
                ref = stack[--sp];
            }
        }
        const int first = leaf_first(ref), cnt = leaf_count(ref);
        for (int i = 0; i < cnt; ++i) {
            int ti = first + i;
            float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
            if (tris_tested) ++*tris_tested;
            float t, u, v;
            if (FAST ? tri_test_fast(o, d, g0, g1, g2, limit, t, u, v) : tri_test(o, d, g0, g1, g2, limit, t, u, v)) return true;
        }
        if (sp == 0) return false;
        ref = stack[--sp];
    }
}

// ------------------------------------------------------------------ the fast walk (trav=1)
// Bound by the L1's data pipe and by issue slots at once (first-bounce shadow
// rays: 84 % of the L1's wavefronts and 64 % of the issue slots), so a node
// visit takes few, wide instructions: two 32-byte loads instead of four of
// 16, six two-wide FMAs for the twelve quotients (three-operand min and max
// the compiler forms by itself too).
// 1M-triangle frame of 1080p x 64 spp against four 16-byte loads and scalar
// FMAs: closest hit 78.2 -> 73.2 ms, shadow rays 46.3 -> 42.9, L1 wavefronts
// of the first shadow bounce 333 M -> 284 M, warp instructions 982 M -> 835 M.
// Two FMAs in one instruction (each rounded as __fmaf_rn).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
        " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// 32 bytes in one load (p 32-byte aligned, read-only data).
struct f8 {
    float v[8];
};
__device__ __forceinline__ f8 ld8(const void* p) {
    f8 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
        : "l"(p));
    return r;
}

// A ray's reciprocals and -o r (make_slab_ray's values) in the pairs of a
// FastNode child.
struct FastRay {
    float2 rxy, rzz, cxy, czz;
};
__device__ __forceinline__ FastRay make_fast_ray(const SlabRay& r) {
    return {make_float2(r.rx, r.ry), make_float2(r.rz, r.rz), make_float2(r.cx, r.cy), make_float2(r.cz, r.cz)};
}

// The one-FMA test alone, on boxes widened on the host: each bound is moved
// outward by more than the error of these quotients and of the reference's
// own rounding for every ray origin within DeviceScene::fast_origin_bound, so
// the test accepts every box the exact test accepts for the unwidened box
// (and a sliver more around it) without a margin or a fallback. The pruning
// limit is folded in: a box is kept when max(entry, 0) <= min(exit, lim),
// 0 <= lim <= 1e18. te receives max(entry, 0). A child's box lies inside its
// parent's and fma(b, r, c) is monotone in b, so a leaf is reached exactly
// when its own box passes.
__device__ __forceinline__ bool fast_box(const FastRay& R, const f8& b, float lim, float& te) {
    const float2 l = fma2(make_float2(b.v[0], b.v[1]), R.rxy, R.cxy);
    const float2 h = fma2(make_float2(b.v[2], b.v[3]), R.rxy, R.cxy);
    const float2 z = fma2(make_float2(b.v[4], b.v[5]), R.rzz, R.czz);
    te = fmaxf(max3(fminf(l.x, h.x), fminf(l.y, h.y), fminf(z.x, z.y)), 0.0f);
    return te <= fminf(min3(fmaxf(l.x, h.x), fmaxf(l.y, h.y), fmaxf(z.x, z.y)), lim);
}

// Closest hit on the widened boxes: the loop and the rules of
// closest_hit_ww, triangles by the fast test with its exact fallback.
// POSTPONE: a lane's first leaf waits until every lane of the warp has one,
// else each lane tests a leaf when it reaches it. The biased determinant lets
// some tiny triangles report a t short of their box, and for those the order
// of leaf and node decides; without postponing it depends on the ray alone, so
// rays may be regrouped (sorted rays, 1080p x 64 spp: 61.8 ms with postponed
// leaves, 64.9 without, but an occasional path that ends elsewhere).
template <bool POSTPONE>
__device__ __forceinline__ int closest_hit_fast(const DeviceScene& S, f3 o, f3 d, float& best_t, float& best_b1,
                                                float& best_b2, uint32_t* nodes_visited = nullptr,
                                                uint32_t* tris_tested = nullptr) {
    best_t = 1e18f; best_b1 = 0.f; best_b2 = 0.f;
    int best = -1, best_leaf = -1;
    if (S.root_ref == INT32_MIN) return -1;
    const SlabRay Q = make_slab_ray(o, d);
    float te;
    if (!box_test(Q, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return -1;
    const FastRay R = make_fast_ray(Q);
    int2 stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    auto pop = [&]() {
        while (sp > 0) {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) <= best_t * S.prune_k) return e.x;
        }
        return (int)NR_TRAV_END;
    };
    int leaf = 0;  // postponed leaf (< 0), or none (>= 0)
    if (ref < 0) { leaf = ref; ref = NR_TRAV_END; }  // the whole scene is one leaf
    while (ref != NR_TRAV_END || leaf < 0) {
        while ((unsigned)ref < (unsigned)NR_TRAV_END) {
            const FastNode& N = S.nodes_fast[ref];
            const f8 a = ld8(N.c0), b = ld8(N.c1);
            if (nodes_visited) ++*nodes_visited;
            const float lim = fminf(best_t * S.prune_k, 1e18f);
            float t0, t1;
            const bool h0 = fast_box(R, a, lim, t0), h1 = fast_box(R, b, lim, t1);
            const int k0 = __float_as_int(a.v[6]), k1 = __float_as_int(a.v[7]);
            if (h0 && h1) {
                int nr = k0, fr = k1;
                float ft = t1;
                if (t1 < t0) { nr = k1; fr = k0; ft = t0; }
                stack[sp++] = make_int2(fr, __float_as_int(ft));
                ref = nr;
            } else if (h0) {
                ref = k0;
            } else if (h1) {
                ref = k1;
            } else {
                ref = pop();
            }
            if (POSTPONE) {
                if (ref < 0 && leaf >= 0) { leaf = ref; ref = pop(); }
                if (!__any_sync(__activemask(), leaf >= 0)) break;
            }
        }
        if (!POSTPONE && ref < 0) { leaf = ref; ref = 0; }
        while (leaf < 0) {
            const int first = leaf_first(leaf), cnt = leaf_count(leaf);
            float lt = 1e18f;
            int li = -1;
            for (int i = 0; i < cnt; ++i) {
                const int ti = first + i;
                const float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
                if (tris_tested) ++*tris_tested;
                float tt, u, v;
                // t < lt within the leaf, and t <= best_t (a tie with the best
                // so far still decides by leaf order): the next float above
                // best_t as the limit rejects farther hits before the exact
                // quotients
                const float cap = fminf(lt, __uint_as_float(__float_as_uint(best_t) + 1u));
                if (tri_test_fast(o, d, g0, g1, g2, cap, tt, u, v)) { lt = tt; li = ti; }
            }
            if (li >= 0 && (lt < best_t || (lt == best_t && first > best_leaf))) {
                best_t = lt; best = li; best_leaf = first;
            }
            if (POSTPONE) {
                leaf = ref;
                if (ref < 0) ref = pop();
            } else {
                leaf = 0;
                ref = pop();
            }
        }
    }
    if (best >= 0) {
        const float4 g0 = __ldg(&S.tri_geo[3 * best]), g1 = __ldg(&S.tri_geo[3 * best + 1]), g2 = __ldg(&S.tri_geo[3 * best + 2]);
        float t;
        tri_test(o, d, g0, g1, g2, 3.0e38f, t, best_b1, best_b2);
    }
    return best;
}

// The nearest hit among a leaf's triangles with t <= best_t (a tie with the
// best so far is decided by leaf order): its triangle and t, or -1. The next
// float above best_t as the limit rejects farther hits before the exact
// quotients.
__device__ __forceinline__ int leaf_hit(const DeviceScene& S, f3 o, f3 d, int first, int cnt, float best_t, float& lt) {
    int li = -1;
    lt = 1e18f;
    for (int i = 0; i < cnt; ++i) {
        const int ti = first + i;
        const float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
        float t, u, v;
        const float cap = fminf(lt, __uint_as_float(__float_as_uint(best_t) + 1u));
        if (tri_test_fast(o, d, g0, g1, g2, cap, t, u, v)) { lt = t; li = ti; }
    }
    return li;
}
// Whether the reference's test enters the box of the leaf that starts at
// triangle `first`, no later than lim. Exact boxes nest and the exact
// quotients are monotone in the bounds, so that is the reference's reach
// whatever stands above the leaf.
__device__ __forceinline__ bool leaf_reached(const DeviceScene& S, f3 o, f3 d, int first, float lim) {
    const int at = __float_as_int(__ldg(&S.tri_geo[3 * first + 2]).w);  // parent and side; -1: the root
    if (at < 0) return true;
    const GpuNode& N = S.nodes[at >> 1];
    const float4 xy = __ldg(at & 1 ? &N.b : &N.a), z = __ldg(&N.c);
    float te;
    return box_test(make_slab_ray(o, d), xy.x, xy.y, xy.z, xy.w, at & 1 ? z.z : z.x, at & 1 ? z.w : z.y, te) && te <= lim;
}
// The winner's barycentrics, recomputed rather than carried through the walk:
// both triangle tests return the correctly rounded quotients.
__device__ __forceinline__ void hit_barycentrics(const DeviceScene& S, f3 o, f3 d, int tri, float& b1, float& b2) {
    const float4 g0 = __ldg(&S.tri_geo[3 * tri]), g1 = __ldg(&S.tri_geo[3 * tri + 1]), g2 = __ldg(&S.tri_geo[3 * tri + 2]);
    float t;
    tri_test(o, d, g0, g1, g2, 3.0e38f, t, b1, b2);
}

// closest_hit's answer by the widened boxes: its order (near first, a leaf at
// once), its pruning, and its reach: a leaf the widened boxes reach counts
// only if its exact box passes too, checked where one of its triangles is
// hit. For origins within S.fast_origin_bound.
__device__ __forceinline__ int closest_hit_query(const DeviceScene& S, f3 o, f3 d, float& best_t, float& best_b1,
                                                 float& best_b2) {
    best_t = 1e18f; best_b1 = 0.f; best_b2 = 0.f;
    int best = -1, best_leaf = -1;
    if (S.root_ref == INT32_MIN) return -1;
    {
        const SlabRay Q = make_slab_ray(o, d);
        float te;
        if (!box_test(Q, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return -1;
    }
    const FastRay R = make_fast_ray(make_slab_ray(o, d));
    int2 stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    auto pop = [&]() {
        while (sp > 0) {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) <= best_t * S.prune_k) return e.x;
        }
        return (int)NR_TRAV_END;
    };
    while (ref != NR_TRAV_END) {
        while ((unsigned)ref < (unsigned)NR_TRAV_END) {
            const FastNode& N = S.nodes_fast[ref];
            const f8 a = ld8(N.c0), b = ld8(N.c1);
            const float lim = fminf(best_t * S.prune_k, 1e18f);
            float t0, t1;
            const bool h0 = fast_box(R, a, lim, t0), h1 = fast_box(R, b, lim, t1);
            const int k0 = __float_as_int(a.v[6]), k1 = __float_as_int(a.v[7]);
            if (h0 && h1) {
                int nr = k0, fr = k1;
                float ft = t1;
                if (t1 < t0) { nr = k1; fr = k0; ft = t0; }
                stack[sp++] = make_int2(fr, __float_as_int(ft));
                ref = nr;
            } else if (h0) {
                ref = k0;
            } else if (h1) {
                ref = k1;
            } else {
                ref = pop();
            }
        }
        if (ref == NR_TRAV_END) break;
        const int first = leaf_first(ref);
        float lt;
        const int li = leaf_hit(S, o, d, first, leaf_count(ref), best_t, lt);
        if (li >= 0 && (lt < best_t || (lt == best_t && first > best_leaf)) && leaf_reached(S, o, d, first, best_t * S.prune_k)) {
            best_t = lt; best = li; best_leaf = first;
        }
        ref = pop();
    }
    if (best >= 0) hit_barycentrics(S, o, d, best, best_b1, best_b2);
    return best;
}

// ------------------------------------------------------------------ the four-wide walk
// For few rays: each walks alone, one dependent load after the other, and
// takes half the steps through nodes of up to four children (build_wide). us:
// 3072 paths to their end 227 -> 178, 15,360 289 -> 240, 129,600 547 -> 511;
// 65,536 camera rays 123 -> 108. Many rays are bound by the L1's bandwidth
// and the issue slots instead, where a visit of 112 bytes and a sort of four
// gains nothing (518,400 paths 1346 -> 1361; 1080p x 64 spp 136 -> 147 ms).

// A ray prepared for WideNode: per axis make_slab_ray's values and the byte
// offset in a node of the planes it meets first; the far planes are at that ^ 16.
struct WideRay {
    float rx, ry, rz, cx, cy, cz;
    uint32_t sx, sy, sz;
};
__device__ __forceinline__ WideRay make_wide_ray(const SlabRay& s) {
    WideRay r;
    r.rx = s.rx; r.ry = s.ry; r.rz = s.rz;
    r.cx = s.cx; r.cy = s.cy; r.cz = s.cz;
    r.sx = (__float_as_uint(s.rx) >> 27) & 16u;
    r.sy = 32u + ((__float_as_uint(s.ry) >> 27) & 16u);
    r.sz = 64u + ((__float_as_uint(s.rz) >> 27) & 16u);
    return r;
}

// fast_box for the four children of a node: entry distances and whether each
// is entered. fma(b, r, c) is monotone in b, so the planes taken by the sign
// of r give the smaller and larger quotient.
__device__ __forceinline__ void wide_test(const DeviceScene& S, const WideRay& R, int ref, float lim, float (&t)[4],
                                          bool (&h)[4], int4& kids) {
    const char* base = reinterpret_cast<const char*>(S.wide);
    const uint32_t off = (uint32_t)ref * (uint32_t)sizeof(WideNode);
    const uint32_t ox = off + R.sx, oy = off + R.sy, oz = off + R.sz;
    auto ld = [&](uint32_t at) { return __ldg(reinterpret_cast<const float4*>(base + at)); };
    const float4 nx = ld(ox), fx = ld(ox ^ 16u), ny = ld(oy), fy = ld(oy ^ 16u), nz = ld(oz), fz = ld(oz ^ 16u);
    kids = __ldg(reinterpret_cast<const int4*>(base + off + 96u));
    const float2 rx = make_float2(R.rx, R.rx), ry = make_float2(R.ry, R.ry), rz = make_float2(R.rz, R.rz);
    const float2 cx = make_float2(R.cx, R.cx), cy = make_float2(R.cy, R.cy), cz = make_float2(R.cz, R.cz);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        auto half = [&](float4 v) { return p ? make_float2(v.z, v.w) : make_float2(v.x, v.y); };
        const float2 ax = fma2(half(nx), rx, cx), ay = fma2(half(ny), ry, cy), az = fma2(half(nz), rz, cz);
        const float2 bx = fma2(half(fx), rx, cx), by = fma2(half(fy), ry, cy), bz = fma2(half(fz), rz, cz);
        t[2 * p] = fmaxf(max3(ax.x, ay.x, az.x), 0.0f);
        t[2 * p + 1] = fmaxf(max3(ax.y, ay.y, az.y), 0.0f);
        h[2 * p] = t[2 * p] <= fminf(min3(bx.x, by.x, bz.x), lim);
        h[2 * p + 1] = t[2 * p + 1] <= fminf(min3(bx.y, by.y, bz.y), lim);
    }
}

// Puts the child that comes first of two in a: the nearer, or with FAR the farther.
template <bool FAR>
__device__ __forceinline__ void wide_order(float& ta, int& ra, float& tb, int& rb) {
    const bool s = FAR ? tb > ta : tb < ta;
    const float t0 = s ? tb : ta, t1 = s ? ta : tb;
    const int r0 = s ? rb : ra, r1 = s ? ra : rb;
    ta = t0; tb = t1; ra = r0; rb = r1;
}

// Closest hit, nearest child first, a leaf at once. EXACT: leaves count by
// their exact boxes (closest_hit_query's answer), else by the widened ones.
// The host bounds the stack this needs, whatever the ray (wide_tree).
template <bool EXACT>
__device__ __forceinline__ int closest_hit_wide(const DeviceScene& S, f3 o, f3 d, float& best_t, float& best_b1,
                                                float& best_b2) {
    best_t = 1e18f; best_b1 = 0.f; best_b2 = 0.f;
    int best = -1, best_leaf = -1;
    if (S.root_ref == INT32_MIN) return -1;
    {
        const SlabRay Q = make_slab_ray(o, d);
        float te;
        if (!box_test(Q, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return -1;
    }
    const WideRay R = make_wide_ray(make_slab_ray(o, d));
    const float none = __int_as_float(0x7f800000);
    int2 stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    auto pop = [&]() {
        while (sp > 0) {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) <= best_t * S.prune_k) return e.x;
        }
        return (int)NR_TRAV_END;
    };
    while (ref != NR_TRAV_END) {
        while ((unsigned)ref < (unsigned)NR_TRAV_END) {
            float t[4];
            bool h[4];
            int4 k;
            wide_test(S, R, ref, fminf(best_t * S.prune_k, 1e18f), t, h, k);
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = h[i] ? t[i] : none;
            wide_order<false>(t[0], k.x, t[1], k.y);
            wide_order<false>(t[2], k.z, t[3], k.w);
            wide_order<false>(t[0], k.x, t[2], k.z);
            wide_order<false>(t[1], k.y, t[3], k.w);
            wide_order<false>(t[1], k.y, t[2], k.z);
            if (t[3] < none) stack[sp++] = make_int2(k.w, __float_as_int(t[3]));
            if (t[2] < none) stack[sp++] = make_int2(k.z, __float_as_int(t[2]));
            if (t[1] < none) stack[sp++] = make_int2(k.y, __float_as_int(t[1]));
            ref = t[0] < none ? k.x : pop();
        }
        if (ref == NR_TRAV_END) break;
        const int first = leaf_first(ref);
        float lt;
        const int li = leaf_hit(S, o, d, first, leaf_count(ref), best_t, lt);
        if (li >= 0 && (lt < best_t || (lt == best_t && first > best_leaf)) &&
            (!EXACT || leaf_reached(S, o, d, first, best_t * S.prune_k))) {
            best_t = lt; best = li; best_leaf = first;
        }
        ref = pop();
    }
    if (best >= 0) hit_barycentrics(S, o, d, best, best_b1, best_b2);
    return best;
}

// Any hit with t <= tmax, the farthest child first (any_hit_fast's answer).
__device__ __forceinline__ bool any_hit_wide(const DeviceScene& S, f3 o, f3 d, float tmax) {
    if (S.root_ref == INT32_MIN) return false;
    const SlabRay Q = make_slab_ray(o, d);
    float te;
    if (!box_test(Q, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return false;
    const WideRay R = make_wide_ray(Q);
    const float lim = fminf(tmax * S.prune_k, 1e18f);
    const float limit = fminf(1e18f, __uint_as_float(__float_as_uint(tmax) + 1u));  // accepts t <= tmax
    int stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    while (true) {
        while (ref >= 0) {
            float t[4];
            bool h[4];
            int4 k;
            wide_test(S, R, ref, lim, t, h, k);
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = h[i] ? t[i] : -1.f;
            wide_order<true>(t[0], k.x, t[1], k.y);
            wide_order<true>(t[2], k.z, t[3], k.w);
            wide_order<true>(t[0], k.x, t[2], k.z);
            if (t[3] >= 0.f) stack[sp++] = k.w;
            if (t[2] >= 0.f) stack[sp++] = k.z;
            if (t[1] >= 0.f) stack[sp++] = k.y;
            if (t[0] >= 0.f) ref = k.x;
            else if (sp == 0) return false;
            else ref = stack[--sp];
        }
        const int first = leaf_first(ref), cnt = leaf_count(ref);
        for (int i = 0; i < cnt; ++i) {
            const int ti = first + i;
            const float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
            float tt, u, v;
            if (tri_test_fast(o, d, g0, g1, g2, limit, tt, u, v)) return true;
        }
        if (sp == 0) return false;
        ref = stack[--sp];
    }
}

// One ray of nr_intersect: closest_hit's answer by the faster walk where it
// holds, the four-wide one if S has its nodes and the call asks for it. Far
// origins, and directions that are no numbers or beyond 1e30 (their
// reciprocals near the denormals, where the widened boxes' margin is not shown
// to cover the rounding), walk by closest_hit itself.
template <bool WIDE>
__device__ __forceinline__ int query_hit(const DeviceScene& S, f3 o, f3 d, float& t, float& b1, float& b2, uint32_t* err) {
    const float B = S.fast_origin_bound;
    if (fabsf(o.x) <= B && fabsf(o.y) <= B && fabsf(o.z) <= B && fabsf(d.x) <= 1e30f && fabsf(d.y) <= 1e30f && fabsf(d.z) <= 1e30f)
        return WIDE ? closest_hit_wide<true>(S, o, d, t, b1, b2) : closest_hit_query(S, o, d, t, b1, b2);
    return closest_hit(S, o, d, t, b1, b2, err);
}

// Any hit with t <= tmax on the widened boxes, as any_hit_ww. Child order
// (1M-triangle frame, Mpaths/s): far first 759.8, near first 722.5.
__device__ __forceinline__ bool any_hit_fast(const DeviceScene& S, f3 o, f3 d, float tmax,
                                             uint32_t* nodes_visited = nullptr, uint32_t* tris_tested = nullptr) {
    if (S.root_ref == INT32_MIN) return false;
    const SlabRay Q = make_slab_ray(o, d);
    float te;
    if (!box_test(Q, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return false;
    const FastRay R = make_fast_ray(Q);
    const float lim = fminf(tmax * S.prune_k, 1e18f);
    const float limit = fminf(1e18f, __uint_as_float(__float_as_uint(tmax) + 1u));  // accepts t <= tmax
    int stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    while (true) {
        while (ref >= 0) {
            const FastNode& N = S.nodes_fast[ref];
            const f8 a = ld8(N.c0), b = ld8(N.c1);
            if (nodes_visited) ++*nodes_visited;
            float t0, t1;
            const bool h0 = fast_box(R, a, lim, t0), h1 = fast_box(R, b, lim, t1);
            const int k0 = __float_as_int(a.v[6]), k1 = __float_as_int(a.v[7]);
            if (h0 && h1) {
                int nr = k0, fr = k1;
                if (t1 > t0) { nr = k1; fr = k0; }
                stack[sp++] = fr;
                ref = nr;
            } else if (h0) {
                ref = k0;
            } else if (h1) {
                ref = k1;
            } else {
                if (sp == 0) return false;
                ref = stack[--sp];
            }
        }
        const int first = leaf_first(ref), cnt = leaf_count(ref);
        for (int i = 0; i < cnt; ++i) {
            const int ti = first + i;
            const float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
            if (tris_tested) ++*tris_tested;
            float tt, u, v;
            if (tri_test_fast(o, d, g0, g1, g2, limit, tt, u, v)) return true;
        }
        if (sp == 0) return false;
        ref = stack[--sp];
    }
}
template <bool FAST = true>
__device__ __forceinline__ bool any_hit(const DeviceScene& S, f3 o, f3 d, float tmax, uint32_t* err,
                                        uint32_t* nodes_visited = nullptr, uint32_t* tris_tested = nullptr) {
    if (S.root_ref == INT32_MIN) return false;
    SlabRay R = make_slab_ray(o, d);
    float te;
    if (!box_test(R, S.root_lo[0], S.root_hi[0], S.root_lo[1], S.root_hi[1], S.root_lo[2], S.root_hi[2], te)) return false;
    const float lim = tmax * S.prune_k;
    int stack[NR_STACK];
    int sp = 0;
    int ref = S.root_ref;
    const float limit = fminf(1e18f, __uint_as_float(__float_as_uint(tmax) + 1u));  // accepts t <= tmax
    int budget = 2 * S.num_nodes + 8;
    while (true) {
        if (--budget < 0) { atomicOr(err, 2u); return false; }
        if (ref >= 0) {
            const GpuNode& N = S.nodes[ref];
            float4 a = __ldg(&N.a), b = __ldg(&N.b), c = __ldg(&N.c);
            int4 k = __ldg(&N.d);
            if (nodes_visited) ++*nodes_visited;
            float t0, t1;
            bool h0 = (FAST ? box_test_fast(R, a.x, a.y, a.z, a.w, c.x, c.y, t0) : box_test(R, a.x, a.y, a.z, a.w, c.x, c.y, t0)) && t0 <= lim;
            bool h1 = (FAST ? box_test_fast(R, b.x, b.y, b.z, b.w, c.z, c.w, t1) : box_test(R, b.x, b.y, b.z, b.w, c.z, c.w, t1)) && t1 <= lim;
            if (h0 && h1) {
                int nr = k.x, fr = k.y;
                if (t1 < t0) { nr = k.y; fr = k.x; }
                if (sp >= NR_STACK) { atomicOr(err, 1u); return false; }
                stack[sp++] = fr;
                ref = nr;
                continue;
            }
            if (h0) { ref = k.x; continue; }
            if (h1) { ref = k.y; continue; }
        } else {
            int first = leaf_first(ref), cnt = leaf_count(ref);
            for (int i = 0; i < cnt; ++i) {
                int ti = first + i;
                float4 g0 = __ldg(&S.tri_geo[3 * ti]), g1 = __ldg(&S.tri_geo[3 * ti + 1]), g2 = __ldg(&S.tri_geo[3 * ti + 2]);
                if (tris_tested) ++*tris_tested;
                float t, u, v;
                if (FAST ? tri_test_fast(o, d, g0, g1, g2, limit, t, u, v) : tri_test(o, d, g0, g1, g2, limit, t, u, v)) return true;
            }
        }
        if (sp == 0) break;
        ref = stack[--sp];
    }
    return false;
}

}  // namespace nr

