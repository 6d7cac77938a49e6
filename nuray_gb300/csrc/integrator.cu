// The ptnee wavefront: ray generation, closest-hit traversal with the
// material sort, shading with NEE / MIS / Russian roulette, shadow
// traversal, film accumulation. One path per (pixel, sample); its random
// numbers come from a Philox stream keyed by (pixel, sample) so any batch
// split and any thread order give the same image.
//
// Per path and vertex this is RendererPTLS::trace
// (src/renderer/rendererptls.cpp:13-94) unrolled into an iteration:
//   L += T * (NEE term);  T *= |wi.n| f / pdf / prr;  emitter hit: L += T * Ke * fac
// which is the reference's recursion result = NEE + Li * |wi.n| f / pdf / prr.
#include <algorithm>

#include "nr_material.cuh"
#include "integrator.h"
#include "ray_sort.cuh"

namespace nr {

// Warp-aggregated append: every active lane with `want` gets a unique index
// in the queue behind *counter; one atomic per warp.
__device__ __forceinline__ int warp_append(bool want, uint32_t* counter) {
    unsigned active = __activemask();
    unsigned m = __ballot_sync(active, want);
    if (!want) return -1;
    int lane = threadIdx.x & 31;
    int leader = __ffs(m) - 1;
    int rank = __popc(m & ((1u << lane) - 1u));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(m, base, leader);
    return (int)(base + rank);
}

// Append keyed by a small category: lanes sharing a key share one atomic.
__device__ __forceinline__ int warp_append_keyed(int key, uint32_t* counters) {
    unsigned active = __activemask();
    unsigned m = __match_any_sync(active, key);
    int lane = threadIdx.x & 31;
    int leader = __ffs(m) - 1;
    int rank = __popc(m & ((1u << lane) - 1u));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&counters[key], (uint32_t)__popc(m));
    base = __shfl_sync(m, base, leader);
    return (int)(base + rank);
}

// ---------------------------------------------------------------- ray generation
// RendererPTLS::render per-sample body (src/renderer/rendererptls.cpp:170-173):
// jitter x, jitter y, Camera::generateRay.
__global__ void k_raygen(PathState P, WaveDesc W, nr_camera cam, float film_h, Policy pol) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.count) return;
    uint64_t g = W.base + (uint64_t)i;
    uint32_t srel = (uint32_t)(g / (uint64_t)W.npix);
    const uint32_t pidx = (uint32_t)(g % (uint64_t)W.npix);
    int x, y;
    if (W.pix_xy) { x = W.pix_xy[2 * pidx]; y = W.pix_xy[2 * pidx + 1]; }
    else wave_path(W, g, pol.imgw, x, y, srel);
    uint32_t key = (uint32_t)y * (uint32_t)pol.imgw + (uint32_t)x;
    uint32_t sample = W.sample0 + srel;
    Stream s;
    s.init(pol.seed_lo, pol.seed_hi, key, sample, 0);
    float jx = s.next();
    float jy = s.next();
    f3 d = camera_ray(cam, film_h, (float)x + jx, (float)y + jy, (float)pol.imgw, (float)pol.imgh);
    uint32_t flags = pol.force_train ? NR_META_TRAIN : 0u;
    if (pol.coin && (double)s.next() < 0.2) flags = NR_META_TRAIN;  // sampler.random() < 0.2 (renderernrc.cpp:255)
    P.ray_o[i] = make_float4(cam.pos[0], cam.pos[1], cam.pos[2], 0.f);
    P.ray_d[i] = make_float4(d.x, d.y, d.z, 0.f);
    P.thr[i] = make_float4(1.f, 1.f, 1.f, 1.f);
    P.rad[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    P.meta[i] = make_uint4(key, sample, s.n, flags);
    P.queue_in[i] = i;
    if (i == 0) P.counters[CNT_IN] = (uint32_t)W.count;
}

// ---------------------------------------------------------------- closest hit + sort
// Persistent: warps take 32 queue entries at a time from a shared cursor.
// Writes the hit record and buckets the slot by shading category
// (material type of the hit, or CAT_MISS) for the shading pass.
// Adds a per-thread count into a 64-bit device counter, one atomic per warp.
__device__ __forceinline__ void warp_count(uint32_t v, uint32_t* lohi) {
    unsigned long long x = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(reinterpret_cast<unsigned long long*>(lohi), x);
}

// Closest hit, persistent: warps take 32 queue entries at a time from a
// shared cursor, one ray per lane to completion, then the slot is bucketed by
// shading category (material type of the hit, or CAT_MISS).
// trav=1 walks the widened boxes (closest_hit_fast), trav=0 the reference's
// boxes with its exact arithmetic (closest_hit_ww). The
// widened boxes accept every box the exact test accepts, so trav=1 reaches
// every triangle trav=0 reaches (the same hits but where a ray passes within
// about 1e-6 of a box face and hits a triangle there that the exact test's
// rounding excludes). Measured and dropped: refilling idle lanes from the
// queue with separate node and leaf phases, 28 % slower; a four-wide tree of
// these boxes (128-byte nodes, sorted children): half the visits but as many
// L1 wavefronts and more issue slots a visit, 147 against 136 ms a frame; a
// warp walking one shared stack for its 32 shadow rays, 61 against 30 ms even
// on rays sorted by origin and direction.
// Minimum resident 128-thread blocks per SM requested from the register
// allocator for the two traversal kernels. 1M-triangle frame of 1080p x 64
// spp, ms: closest hit at 8 / 10 / 12 blocks 79.2 / 76.6 / 73.2 (40 registers,
// 84 bytes of spills at 12); shadow rays at 8 / 10 / 12 42.7 / 42.9 / 42.5.
// Loop shape: closest hit while-while with postponed leaves, any hit without
// (its first leaf often holds the occluder): 645.4 Mpaths/s against 591.9
// with postponed leaves in both and 606.6 without in either. Also measured
// and dropped for the shadow rays: dynamic fetch of new rays into idle lanes
// (Aila and Laine 2009) at 4, 8 or 16 idle lanes, 571.
#ifndef NR_TRACE_MINB
#define NR_TRACE_MINB 12
#endif
#ifndef NR_SHADOW_MINB
#define NR_SHADOW_MINB 10
#endif
// WALK: 0 exact, 1 fast, both with postponed leaves; 2 fast, 3 exact, whose hits
// do not depend on the warp's other rays (a sorted queue; bounces that the
// adjoint traces twice). Where the order of the paths counts, a sorted queue's
// are bucketed by k_bucket.
template <bool COUNT, int WALK>
__global__ void __launch_bounds__(128, NR_TRACE_MINB) k_trace(PathState P, DeviceScene S, int capacity) {
    const uint32_t n = P.counters[CNT_IN];
    const int lane = threadIdx.x & 31;
    uint32_t nv = 0, nt = 0;
    while (true) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&P.counters[CNT_WORK], 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        uint32_t idx = base + lane;
        if (idx < n) {
            int slot = P.queue_in[idx];
            f3 o = xyz(P.ray_o[slot]), d = xyz(P.ray_d[slot]);
            float t, b1, b2;
            uint32_t *pv = COUNT ? &nv : nullptr, *pt = COUNT ? &nt : nullptr;
            const int tri = WALK == 0   ? closest_hit_ww(S, o, d, t, b1, b2, pv, pt)
                            : WALK == 3 ? closest_hit<false>(S, o, d, t, b1, b2, &P.counters[CNT_ERR], pv, pt)
                                        : closest_hit_fast<WALK == 1>(S, o, d, t, b1, b2, pv, pt);
            P.hit[slot] = make_float4(t, b1, b2, __int_as_float(tri));
            if (P.sort.bucket_after) continue;
            int cat = CAT_MISS;
            if (tri >= 0) cat = S.mats[__float_as_int(__ldg(&S.tri_geo[3 * tri + 1]).w)].type;
            int pos = warp_append_keyed(cat, &P.counters[CNT_CAT]);
            P.sorted[(size_t)cat * capacity + pos] = slot;
        }
    }
    if (COUNT) {
        warp_count(nv, &P.counters[CNT_NODES]);
        warp_count(nt, &P.counters[CNT_TRIS]);
    }
}

// The bucketing of k_trace in the order of the paths, for rays that were traced
// in the order of the ray sort: a cache's training records keep the paths'
// order. Bound by its gathers (the hit triangle's material); one counter update
// per category and 1024 paths. PT+NRC of three steps, 1M triangles, 1080p x 64
// spp: 98.4 ms, against 102.2 with only the shadow rays sorted and 116.5 with
// neither. Waves without that need bucket in k_trace: shading reads slots next to each
// other after k_bucket, but gains what k_bucket costs (122.4 against 123.6 ms).
__global__ void __launch_bounds__(256) k_bucket(PathState P, DeviceScene S, int capacity) {
    __shared__ uint32_t count[NUM_CAT], first[NUM_CAT];
    const uint32_t n = P.counters[CNT_IN];
    for (uint32_t b = blockIdx.x * 1024u; b < n; b += gridDim.x * 1024u) {
        if (threadIdx.x < NUM_CAT) count[threadIdx.x] = 0u;
        __syncthreads();
        int slot[4], cat[4], pos[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t idx = b + 256u * k + threadIdx.x;
            slot[k] = idx < n ? P.sort.queue[idx] : -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cat[k] = CAT_MISS;
            const int tri = slot[k] >= 0 ? __float_as_int(P.hit[slot[k]].w) : -1;
            if (tri >= 0) cat[k] = S.mats[__float_as_int(__ldg(&S.tri_geo[3 * tri + 1]).w)].type;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (slot[k] >= 0) pos[k] = warp_append_keyed(cat[k], count);
        __syncthreads();
        if (threadIdx.x < NUM_CAT && count[threadIdx.x])
            first[threadIdx.x] = atomicAdd(&P.counters[CNT_CAT + threadIdx.x], count[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (slot[k] >= 0) P.sorted[(size_t)cat[k] * capacity + first[cat[k]] + pos[k]] = slot[k];
    }
}

// The sort of k_trace for hits recorded by an earlier pass over the same
// paths (P.hit pointing at that bounce's record): no traversal.
__global__ void k_sort_recorded(PathState P, DeviceScene S, int capacity) {
    const uint32_t n = P.counters[CNT_IN];
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
        const int slot = P.queue_in[idx];
        const int tri = __float_as_int(P.hit[slot].w);
        int cat = CAT_MISS;
        if (tri >= 0) cat = S.mats[__float_as_int(__ldg(&S.tri_geo[3 * tri + 1]).w)].type;
        const int pos = warp_append_keyed(cat, &P.counters[CNT_CAT]);
        P.sorted[(size_t)cat * capacity + pos] = slot;
    }
}

// Shadow rays, persistent like k_trace: occluded when any reachable triangle
// has t <= the ray's limit (any_hit); unoccluded rays add their NEE term.
template <bool COUNT, bool FAST>
__global__ void __launch_bounds__(128, NR_SHADOW_MINB) k_shadow(PathState P, DeviceScene S, float4* t_before) {
    const int32_t* __restrict__ order = P.sort.place[0] ? P.sort.order : nullptr;  // of a sorted queue
    // (a full queue drops rays with an error bit but still counts them)
    const uint32_t n = min(P.counters[CNT_SHADOW], (uint32_t)P.sh_cap);
    const int lane = threadIdx.x & 31;
    uint32_t nv = 0, nt = 0;
    while (true) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&P.counters[CNT_WORK_SH], 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        uint32_t idx = base + lane;
        if (idx < n) {
            if (order) idx = (uint32_t)order[idx];
            float4 o = P.sh_o[idx], d = P.sh_d[idx];
            const bool env = o.w < 0.f;  // an environment sample: k_env_fold adds it
            const float tmax = env ? -o.w : o.w;
            const bool occluded =
                FAST ? any_hit_fast(S, xyz(o), xyz(d), tmax, COUNT ? &nv : nullptr, COUNT ? &nt : nullptr)
                     : any_hit_ww<false>(S, xyz(o), xyz(d), tmax, &P.counters[CNT_ERR], COUNT ? &nv : nullptr,
                                         COUNT ? &nt : nullptr);
            if (P.vis) P.vis[__float_as_int(d.w)] = occluded ? 0 : 1;
            if (env) {
                if (occluded) P.sh_c[idx].x = P.sh_c[idx].y = P.sh_c[idx].z = 0.f;
            } else if (!occluded) {
                int slot = __float_as_int(d.w);
                float4 c = P.sh_c[idx];
                float4 r = P.rad[slot];
                P.rad[slot] = make_float4(r.x + c.x, r.y + c.y, r.z + c.z, 0.f);
                // a cache training record that excludes its vertex's light sample
                const int rec = __float_as_int(c.w);
                if (t_before && rec >= 0) {
                    float4 b = t_before[rec];
                    t_before[rec] = make_float4(b.x + c.x, b.y + c.y, b.z + c.z, 0.f);
                }
            }
        }
    }
    if (COUNT) {
        warp_count(nv, &P.counters[CNT_SH_NODES]);
        warp_count(nt, &P.counters[CNT_SH_TRIS]);
    }
}

// After k_shadow: every environment sample of the bounce adds its
// contribution (zero if occluded) to its path, after the path's area-light
// sample; one environment sample per path, so one writer per slot.
__global__ void k_env_fold(PathState P, float4* t_before) {
    const uint32_t n = min(P.counters[CNT_SHADOW], (uint32_t)P.sh_cap);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
        if (!(P.sh_o[idx].w < 0.f)) continue;
        const int slot = __float_as_int(P.sh_d[idx].w);
        const float4 c = P.sh_c[idx], r = P.rad[slot];
        P.rad[slot] = make_float4(r.x + c.x, r.y + c.y, r.z + c.z, 0.f);
        const int rec = __float_as_int(c.w);
        if (t_before && rec >= 0) {
            const float4 b = t_before[rec];
            t_before[rec] = make_float4(b.x + c.x, b.y + c.y, b.z + c.z, 0.f);
        }
    }
}

// ---------------------------------------------------------------- shading
__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}
// Training paths of the online cache: a fixed hash of (pixel, sample).
__device__ __forceinline__ bool nrc_is_training(uint32_t pixel, uint32_t sample, uint32_t stride) {
    return hash32(pixel ^ hash32(sample + 0x9e3779b9u)) % stride == 0u;
}

// Queues a shadow ray (or, when no hit can come before the limit, adds its
// contribution at once). rec: the training record whose target leaves this
// light sample out, or -1.
// TAIL: trace the shadow ray here (1: exact walk, 2: fast, 3: four-wide)
// instead of queueing it. env: the vertex's environment sample, queued with its limit
// negated: k_shadow leaves its contribution in the queue entry (zero when
// occluded) and k_env_fold adds it after the area-light samples, so each
// path's radiance has one writer at a time and the restatement's order.
template <bool NRC, int TAIL = 0>
__device__ __forceinline__ void emit_shadow(const PathState& P, const DeviceScene& S, const Policy& pol,
                                            const NrcCtx& C, int slot, int rec, f3 so, f3 d, float tmax, f3 c,
                                            uint32_t* shadows, bool env = false) {
    if (TAIL && tmax > 0.f) {
        ++*shadows;
        const bool occluded = TAIL == 3   ? any_hit_wide(S, so, d, tmax)
                              : TAIL == 2 ? any_hit_fast(S, so, d, tmax)
                                          : any_hit_ww<false>(S, so, d, tmax, &P.counters[CNT_ERR]);
        if (occluded) return;
        tmax = 0.f;  // unoccluded: added below
    }
    if (tmax > 0.f) {
        int q = warp_append(true, &P.counters[CNT_SHADOW]);
        if (q >= P.sh_cap) { atomicOr(&P.counters[CNT_ERR], 4u); return; }
        P.sh_o[q] = make_float4(so.x, so.y, so.z, env ? -tmax : tmax);
        P.sh_d[q] = make_float4(d.x, d.y, d.z, __int_as_float(slot));
        P.sh_c[q] = make_float4(c.x, c.y, c.z, __int_as_float(rec));
        if (P.sort.place[0]) ray_place(S, P.sort, 0, (uint32_t)q, so, d);
    } else {
        // c rounded before it is added, as k_shadow adds it from the queue: the
        // same image whichever kernel takes a bounce
        float4 r = P.rad[slot];
        P.rad[slot] = make_float4(radd(r.x, c.x), radd(r.y, c.y), radd(r.z, c.z), 0.f);
        if (NRC && rec >= 0) {
            float4 b = C.t_before[rec];
            C.t_before[rec] = make_float4(radd(b.x, c.x), radd(b.y, c.y), radd(b.z, c.z), 0.f);
        }
    }
}

// MT: the shading category when it is known at compile time (a material
// type, or CAT_MISS), -1 for any. TAIL: light samples traced here (1 by the
// exact walk, 2 by the fast, 3 by the four-wide one) and the continuing path
// not queued. Returns whether the path goes on.
template <bool NRC, int MT = -1, int TAIL = 0>
__device__ __forceinline__ bool shade_one(const PathState& P, const DeviceScene& S, const Policy& pol, int slot,
                                          const NrcCtx& C, uint32_t* shadows = nullptr) {
    float4 h = P.hit[slot];
    float4 thr = P.thr[slot];
    uint4 meta = P.meta[slot];
    const float4 dir4 = P.ray_d[slot];
    f3 dir = xyz(dir4);
    f3 T = xyz(thr);
    int tri = __float_as_int(h.w);
    if (MT == CAT_MISS || (MT < 0 && tri < 0)) {
        if (S.env_tex >= 0) {
            float4 r = P.rad[slot];
            f3 e = env_lookup(S, dir);
            // envis: the previous vertex also sampled the environment; dir4.w
            // holds the BSDF density of this direction (balance heuristic)
            if (dir4.w > 0.f && S.env_weight) e = e * (dir4.w / (dir4.w + env_pdf(S, dir)));
            P.rad[slot] = make_float4(r.x + T.x * e.x, r.y + T.y * e.y, r.z + T.z * e.z, 0.f);
        }
        return false;
    }
    float b1 = h.y, b2 = h.z;
    float4 s0 = __ldg(&S.tri_shade[4 * tri]), s1 = __ldg(&S.tri_shade[4 * tri + 1]);
    float4 s2 = __ldg(&S.tri_shade[4 * tri + 2]), s3 = __ldg(&S.tri_shade[4 * tri + 3]);
    int mat = __float_as_int(s3.w);
    // Triangle::getNormal / getTexCoords (src/scene/triangle.cpp:35-43)
    float w0 = 1.0f - b1 - b2;
    f3 normal = normalized(w0 * xyz(s0) + b1 * xyz(s1) + b2 * xyz(s2));
    f3 wo = -dir;
    const int type = MT >= 0 ? MT : S.mats[mat].type;
    if (type == NR_MAT_LIGHT) {  // emitter: Ke * light_fac (rendererptls.cpp:33-36)
        const nr_material& M = S.mats[mat];
        float4 r = P.rad[slot];
        float lf = thr.w;
        P.rad[slot] = make_float4(r.x + T.x * M.c0[0] * lf, r.y + T.y * M.c0[1] * lf, r.z + T.z * M.c0[2] * lf, 0.f);
        return false;
    }
    // opaque back faces end the path (rendererptls.cpp:41-42)
    if (dot(normal, dir) > 0.f && !mat_transmissive(type)) return false;
    // texture coordinates: t0 = (s0.w, s1.w), t1 = (s2.w, s3.x), t2 = (s3.y, s3.z)
    f3 uv = mk(w0 * s0.w + b1 * s2.w + b2 * s3.y, w0 * s1.w + b1 * s3.x + b2 * s3.z, 0.f);
    MatView M = load_mat(S, mat, uv);
    if (MT >= 0) M.type = MT;  // the switch over material types folds to one case
    f3 o = xyz(P.ray_o[slot]);
    f3 hit_pos = o + dir * h.x;
    Stream rng;
    rng.init(pol.seed_lo, pol.seed_hi, meta.x, meta.y, meta.z);
    float fac = 1.0f;
    const int depth = (int)(meta.w & NR_META_DEPTH_MASK);
    uint32_t flags = meta.w & NR_META_SEEN_DIFFUSE;
    const uint32_t train_flag = meta.w & NR_META_TRAIN;
    bool query_here = false;
    int rec = -1;  // training record whose target leaves out this vertex's light sample
    if (NRC) {
        const bool train = pol.excl ? train_flag != 0 : nrc_is_training(meta.x, meta.y, C.train_stride);
        // Past the first diffuse bounce the cache stands in for the rest of the
        // path: from depth min_depth on, or for training paths from
        // train_depth on (their earlier vertices then learn from it).
        // renderer=nrc asks at any vertex: depth >= path_lim, or
        // path_lim_train on training paths (renderernrc.cpp:130).
        const bool end_here = train ? (C.train_depth > 0 && depth >= C.train_depth) : depth >= C.min_depth;
        const bool diffuse_here = C.first && nrc_diffuse(M, C.rough);
        if ((flags || diffuse_here || pol.excl) && C.query && end_here) {
            int q = warp_append(true, &C.counters[0]);
            C.q_slot[q] = slot;
            C.q_thr[q] = make_float4(T.x, T.y, T.z, 0.f);
            uint32_t qr[8];
            nrc_record(qr, C.lo, C.inv_ext, hit_pos, wo, normal, nrc_roughness(M), M.c0);
            C.q_rec[2 * (size_t)q] = make_uint4(qr[0], qr[1], qr[2], qr[3]);
            C.q_rec[2 * (size_t)q + 1] = make_uint4(qr[4], qr[5], qr[6], qr[7]);
            if (!C.direct) return false;
            query_here = true;  // the light sample below stays explicit
        } else if (train) {
            int r = warp_append(true, &C.counters[1]);
            if (r < C.tcap) {
                C.t_slot[r] = slot;
                C.t_thr[r] = make_float4(T.x, T.y, T.z, 0.f);
                C.t_before[r] = P.rad[slot];
                nrc_encode(reinterpret_cast<uint32_t*>(C.t_x) + (size_t)r * 40, C.lo, C.inv_ext, hit_pos, wo, normal,
                           nrc_roughness(M), M.c0);
                if (C.direct) rec = r;
            }
        }
        if (nrc_diffuse(M, C.rough)) flags = NR_META_SEEN_DIFFUSE;
    }

    // next-event estimation (rendererptls.cpp:49-78)
    if (pol.excl && pol.nee && mat_nee(type)) fac = 0.0f;  // is_light_sampled (renderernrc.cpp:139)
    if (pol.nee && mat_nee(type) && S.num_lights > 0) {
        const int li = pick_light(S, rng.next());
        const float4* L = S.lights + 6 * li;
        float4 l0 = __ldg(&L[0]), l1 = __ldg(&L[1]), l2 = __ldg(&L[2]);
        float4 n0 = __ldg(&L[3]), n1 = __ldg(&L[4]), n2 = __ldg(&L[5]);
        // Triangle::sample (src/scene/triangle.cpp:45-55)
        float r1 = rng.next();
        float r2 = rng.next();
        if (r1 + r2 > 1.f) { r1 = 1.f - r1; r2 = 1.f - r2; }
        float lw = 1.f - r1 - r2;
        f3 light_pos = lw * xyz(l0) + r1 * xyz(l1) + r2 * xyz(l2);
        f3 light_normal = normalized(lw * xyz(n0) + r1 * xyz(n1) + r2 * xyz(n2));
        f3 light_vec = light_pos - hit_pos;
        f3 wl = normalized(light_vec);
        f3 Ke = mk(l0.w, l1.w, l2.w);
        float light_pdf = S.light_p;
        float cos_l = dot(light_normal, -wl);
        float light_omega_pdf = light_pdf * dot(light_vec, light_vec) / smax(1e-6f, cos_l);
        float brdf_omega_pdf = mat_pdf(M, wo, normal, wl);
        float mis = light_omega_pdf / (light_omega_pdf + brdf_omega_pdf);
        if (!pol.mis) mis = 0.5f;
        if (pol.excl) mis = 1.0f;  // renderernrc.cpp:155: no MIS weight
        else fac = 1.0f - mis;
        f3 brdf = mat_bxdf(M, wo, normal, wl);
        f3 Ll = Ke / norm2(light_vec) * smax(0.f, cos_l) / light_pdf;
        const float geo = smax(0.f, dot(normal, normalized(light_pos - hit_pos)));
        f3 c = Ll * brdf * geo * mis;
        c = c * T;
        if (c.x != 0.f || c.y != 0.f || c.z != 0.f || (pol.adj && cos_l > 0.f && geo > 0.f && mis > 0.f)) {
            // Visible iff the closest t satisfies t + 2e-3 > |light_vec| (in
            // double there), i.e. occluded iff some hit has t <= |lv| - 2e-3.
            double lim = (double)norm(light_vec) - 2e-3;
            float tmax = lim > 0.0 ? __double2float_rd(lim) : 0.0f;
            emit_shadow<NRC, TAIL>(P, S, pol, C, slot, rec, hit_pos + wl * 1e-3f, wl, tmax, c, shadows);
        }
    }
    // envis: one environment light sample more (no counterpart in the
    // reference), weighted against the BSDF-sampled miss by the balance
    // heuristic; its two draws follow the area-light draws
    bool env_sampled = false;
    if (pol.envis && pol.nee && mat_nee(type) && S.env_weight) {
        env_sampled = true;
        const float r1 = rng.next(), r2 = rng.next();
        f3 we;
        float pe;
        if (env_sample(S, r1, r2, we, pe)) {
            const float cosn = dot(normal, we);
            if (cosn > 0.f) {
                // at the depth limit no BSDF sample follows: the light sample takes the full weight
                const bool last = pol.maxdepth > 0 && depth + 1 >= pol.maxdepth;
                const float pb = last ? 0.f : mat_pdf(M, wo, normal, we);
                const f3 c = T * mat_bxdf(M, wo, normal, we) * env_lookup(S, we) * (cosn / (pe + pb));
                if (c.x != 0.f || c.y != 0.f || c.z != 0.f)
                    emit_shadow<NRC, TAIL>(P, S, pol, C, slot, rec, hit_pos + we * 1e-3f, we, 3.0e38f, c, shadows, true);
            }
        }
    }
    if (NRC && query_here) return false;
    if (pol.maxdepth > 0 && depth + 1 >= pol.maxdepth) return false;
    // Russian roulette (rendererptls.cpp:80-83)
    float prr = depth < pol.rrdepth ? 1.0f : pol.prr;
    float u = rng.next();
    if (depth >= pol.rrdepth && (pol.excl ? !(u < prr) : u > prr)) return false;  // renderernrc.cpp:162: go on while u < prr
    f3 wi = mat_sample(M, rng, wo, normal);
    float pdf = mat_pdf(M, wo, normal, wi);
    f3 brdf = mat_bxdf(M, wo, normal, wi);
    // contri = Li * |wi.n| * brdf / pdf / prr (rendererptls.cpp:90)
    f3 Tn = T * fabsf(dot(wi, normal)) * brdf / pdf / prr;
    f3 no = hit_pos + wi * 1e-3f;
    if (!TAIL) {
        int q = warp_append(true, &P.counters[CNT_OUT]);
        P.queue_out[q] = slot;
        if (P.sort.place[1]) ray_place(S, P.sort, 1, (uint32_t)q, no, wi);
    }
    P.ray_o[slot] = make_float4(no.x, no.y, no.z, 0.f);
    P.ray_d[slot] = make_float4(wi.x, wi.y, wi.z, env_sampled ? pdf : 0.f);
    P.thr[slot] = make_float4(Tn.x, Tn.y, Tn.z, fac);
    P.meta[slot] = make_uint4(meta.x, meta.y, rng.n, (uint32_t)(depth + 1) | flags | train_flag);
    return true;
}

// Shading: one kernel per shading category of the bucketed queue (the five
// material types, emitters, misses), each compiled with its category fixed
// so the material switch folds to one case and the kernel keeps only that
// material's registers. All seven are launched per bounce; each strides
// over its device-side count with at most 32 rounds of resident blocks.
// Measured on the 1M-triangle frame (Mpaths/s): one kernel for all
// categories 761.6, per category 771.3 (C3, mixed materials: 751.4 ->
// 761.2); 8, 32 or 128 rounds of blocks 769.9, 771.3, (C3) 759.7.
// Blocks per SM asked of the register allocator: 8 (64 registers). For the
// single kernel before: 646.3 uncapped (94 registers), 651.8 at 6, 657.4
// at 8, 647.3 at 10, 629.7 at 12; per category 6 gives 763.3 against 771.3;
// re-checked with the tail kernel and the category mask: 6 / 8 / 10 give
// 766.0 / 773.9 / 768.6.
#ifndef NR_SHADE_MINB
#define NR_SHADE_MINB 8
#endif
#ifndef NR_SHADE_ROUNDS
#define NR_SHADE_ROUNDS 32
#endif
template <bool NRC, int MT>
__global__ void __launch_bounds__(128, NR_SHADE_MINB) k_shade(PathState P, DeviceScene S, Policy pol, int capacity,
                                                              NrcCtx C) {
    if (MT >= 0) {
        const uint32_t n = P.counters[CNT_CAT + (MT >= 0 ? MT : 0)];
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            shade_one<NRC, MT>(P, S, pol, P.sorted[(size_t)MT * capacity + i], C);
        return;
    }
    // MT = -1: every category in one kernel (categories are contiguous, so
    // a warp mostly runs one material's code)
    uint32_t start[NUM_CAT];
    uint32_t total = 0;
#pragma unroll
    for (int c = 0; c < NUM_CAT; ++c) { start[c] = total; total += P.counters[CNT_CAT + c]; }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int c = 0;
#pragma unroll
        for (int k = 1; k < NUM_CAT; ++k) if (i >= start[k]) c = k;
        shade_one<NRC>(P, S, pol, P.sorted[(size_t)c * capacity + (i - start[c])], C);
    }
}
// Bounces of at most SHADE_SPLIT_MIN paths shade with the one kernel for all
// categories: they are short, and six mostly empty launches per bounce cost
// more than the split saves (time to relMSE 1e-3 with 960x540 frames of 1 spp:
// 10.40 s with one kernel, 11.34 s with seven; later bounces of a large wave,
// the room at 640x480 x 16 spp: 5.06 ms with one, 5.22 with five). With the
// cache the wave's size decides, so that its training records keep one order.
template <bool NRC>
static void launch_shade(const PathState& P, const DeviceScene& S, const Policy& pol, int capacity, int paths, int blocks,
                         const NrcCtx& C, cudaStream_t st) {
    if (paths <= SHADE_SPLIT_MIN) {
        k_shade<NRC, -1><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
        return;
    }
    // categories of material types absent from the scene can hold no path
    if (S.cat_mask & (1u << NR_MAT_LAMBERT)) k_shade<NRC, NR_MAT_LAMBERT><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    if (S.cat_mask & (1u << NR_MAT_GGXR)) k_shade<NRC, NR_MAT_GGXR><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    if (S.cat_mask & (1u << NR_MAT_GGX)) k_shade<NRC, NR_MAT_GGX><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    if (S.cat_mask & (1u << NR_MAT_GLASS)) k_shade<NRC, NR_MAT_GLASS><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    if (S.cat_mask & (1u << NR_MAT_BLINNPHONG))
        k_shade<NRC, NR_MAT_BLINNPHONG><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    if (S.cat_mask & (1u << NR_MAT_LIGHT)) k_shade<NRC, NR_MAT_LIGHT><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
    k_shade<NRC, CAT_MISS><<<blocks, 128, 0, st>>>(P, S, pol, capacity, C);
}

// The rest of every live path in one launch, one thread per path: closest
// hit, then shade_one in its TAIL form (light samples traced inline), until
// the path ends. For bounces of few paths (run_waves decides): the wavefront
// waits at each bounce for its slowest ray in each of its kernels, this kernel
// only for the slowest path. Same functions, same results.
#ifndef NR_TAIL_MAX_BOUNCES
#define NR_TAIL_MAX_BOUNCES 4096
#endif
// Resident blocks per SM requested for the tail kernel. Its paths wait on
// dependent traversal loads with few live lanes, so warps in flight pay more
// than the registers' spills cost: 960x540 frames of 1 spp take 1.16 ms at 8
// (64 registers) and 9 blocks; with a path per thread to its end 1.543 at 4 (89
// registers), 1.536 at 6, 1.463 at 8, 1.459 at 10, 1.476 at 12 and 1.535 at 16.
#ifndef NR_TAIL_MINB
#define NR_TAIL_MINB 8
#endif
// With the four-wide walk (few paths) the registers pay more: 3072 paths 181
// us at 8 blocks, 178 at 6; 57,600 365 / 354; 522,240 of every material (about
// half of them live at the tail) 730 / 716.
#define NR_TAIL_MINB_WIDE 6
// Paths a warp starts with: a warp walks for as long as its slowest ray in
// every phase, so a few paths are spread over 16 warps per SM, and up to 8 warps
// per SM before warps fill (a path per thread, 1M triangles, 3072 paths: 350 us
// with full warps, 263 / 238 / 227 / 214 over 4 / 8 / 16 / 32 warps per SM;
// 15,360 paths 354 / 314 / 289 / 315; the room of 36 triangles, bound by issue
// slots at 61,440 paths: 510 / 509 / 570 / 633).
#define NR_TAIL_WARPS 16
__host__ __device__ inline uint32_t tail_paths_per_warp(uint32_t n, uint32_t sms) {
    const uint32_t wide = sms * NR_TAIL_WARPS, warps = n <= 8u * wide ? wide : wide / 2u;
    const uint32_t take = (n + warps - 1u) / warps;
    return take < 1u ? 1u : (take > 32u ? 32u : take);
}
// WALK: 1 exact, 2 fast, 3 four-wide. A lane whose path has ended takes the
// next one of the queue at once (a warp's 32 paths are not done before the
// longest of them, and most end early: 518,400 paths 1346 us with a path per
// thread, 1175 with refilled lanes; refilled once 8 / 16 / 32 lanes are idle
// 1180 / 1197 / 1296).
template <bool NRC, int WALK>
__global__ void __launch_bounds__(128, WALK == 3 ? NR_TAIL_MINB_WIDE : NR_TAIL_MINB) k_tail(PathState P, DeviceScene S, Policy pol,
                                                                                              NrcCtx C, uint32_t sms) {
    const uint32_t n = P.counters[CNT_IN], take = tail_paths_per_warp(n, sms);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), lane = threadIdx.x & 31u;
    const uint32_t first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * take + lane;
    const uint32_t given = warps * take;  // paths the warps start with; the rest are taken as lanes fall idle
    bool more = given < n;                // (uniform) whether there may be any left
    int slot = lane < take && first < n ? P.queue_in[first] : -1;
    int b = 0;
    uint32_t rays = 0, shadows = 0;
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, slot < 0);
        if (more && idle) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&P.counters[CNT_WORK], (uint32_t)__popc(idle));
            base = given + __shfl_sync(0xffffffffu, base, 0);
            more = base + (uint32_t)__popc(idle) < n;
            if (slot < 0) {
                const uint32_t i = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (i < n) { slot = P.queue_in[i]; b = 0; }
            }
        }
        if (!__any_sync(0xffffffffu, slot >= 0)) break;
        if (slot >= 0) {
            const f3 o = xyz(P.ray_o[slot]), d = xyz(P.ray_d[slot]);
            float t, b1, b2;
            const int tri = WALK == 3   ? closest_hit_wide<false>(S, o, d, t, b1, b2)
                            : WALK == 2 ? closest_hit_fast<false>(S, o, d, t, b1, b2)
                                        : closest_hit_ww(S, o, d, t, b1, b2);
            P.hit[slot] = make_float4(t, b1, b2, __int_as_float(tri));
            ++rays;
            bool on = shade_one<NRC, -1, WALK>(P, S, pol, slot, C, &shadows);
            if (on && ++b >= NR_TAIL_MAX_BOUNCES) {  // bounce cap: the path did not end
                atomicOr(&P.counters[CNT_ERR], (uint32_t)NR_ERRBIT_BOUNCES);
                on = false;
            }
            if (!on) slot = -1;
        }
        __syncwarp();
    }
    warp_count(rays, &P.counters[CNT_RAYS]);
    warp_count(shadows, &P.counters[CNT_SHRAYS]);
}

// The two queues of a sorted bounce: blockIdx.y 0 writes the order of the
// shadow queue, 1 the continuing paths into queue_out. Bound by its scattered
// four-byte writes (132.7M paths' first bounce 3.6 ms); four entries a thread
// and 32 blocks per SM in flight: 64 spp 123.7 ms, 124.0 with one entry and 4
// blocks, 16 spp 32.67 / 32.76.
constexpr int ORDER_ENTRIES = 4, ORDER_BLOCKS = 32;
__global__ void __launch_bounds__(256) k_ray_order(PathState P) {
    const int which = blockIdx.y;
    const uint32_t n = which ? P.counters[CNT_OUT] : min(P.counters[CNT_SHADOW], (uint32_t)P.sh_cap);
    int32_t* __restrict__ to = which ? P.queue_out : P.sort.order;
    const uint2* __restrict__ place = P.sort.place[which];
    const int32_t* __restrict__ queue = which ? P.sort.queue : nullptr;
    for (uint32_t b = blockIdx.x * (256u * ORDER_ENTRIES); b < n; b += gridDim.x * (256u * ORDER_ENTRIES)) {
        uint2 a[ORDER_ENTRIES];
        uint32_t at[ORDER_ENTRIES];
        int32_t e[ORDER_ENTRIES];
#pragma unroll
        for (int k = 0; k < ORDER_ENTRIES; ++k) {
            const uint32_t q = b + 256u * k + threadIdx.x;
            a[k] = q < n ? __ldcs(place + q) : make_uint2(0u, 0u);
            e[k] = queue && q < n ? __ldcs(queue + q) : (int32_t)q;
        }
#pragma unroll
        for (int k = 0; k < ORDER_ENTRIES; ++k) at[k] = ray_offset(P.sort, which, a[k]);
#pragma unroll
        for (int k = 0; k < ORDER_ENTRIES; ++k)
            if (b + 256u * k + threadIdx.x < n) to[at[k]] = e[k];
    }
}

// ---------------------------------------------------------------- shadow rays
// Moves the continuation queue into place for the next bounce and clears the
// per-bounce counters; also keeps the 64-bit ray totals.
__global__ void k_advance(uint32_t* counters) {
    uint32_t in = counters[CNT_IN], sh = counters[CNT_SHADOW];
    unsigned long long* rays = reinterpret_cast<unsigned long long*>(counters + CNT_RAYS);
    unsigned long long* shr = reinterpret_cast<unsigned long long*>(counters + CNT_SHRAYS);
    *rays += in;
    *shr += sh;
    counters[CNT_IN] = counters[CNT_OUT];
    counters[CNT_OUT] = 0;
    counters[CNT_SHADOW] = 0;
    counters[CNT_WORK] = 0;
    counters[CNT_WORK_SH] = 0;
    for (int c = 0; c < NUM_CAT; ++c) counters[CNT_CAT + c] = 0;
}

// Clears the per-wave counters; the error word and the totals from
// CNT_RAYS on are kept for the whole render.
__global__ void k_reset_counters(uint32_t* counters) {
    int i = threadIdx.x;
    if (i < CNT_RAYS && i != CNT_ERR) counters[i] = 0;
}

// ---------------------------------------------------------------- film
// For every pixel of the wave, adds max(0, L) of its samples in sample order
// (rendererptls.cpp:173). film holds npix float4 sums.
__global__ void k_film(PathState P, WaveDesc W, float4* film, int imgw) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)W.npix) return;
    int x, y;
    const uint64_t end = W.base + (uint64_t)W.count;
    if (W.tiled == 2) {
        const uint32_t tp = (uint32_t)(W.g_w * W.g_h), tile = p / tp, tiles_x = (uint32_t)imgw / (uint32_t)W.g_w;
        x = (int)((tile % tiles_x) * (uint32_t)W.g_w + (p % tp) % (uint32_t)W.g_w);
        y = (int)((tile / tiles_x) * (uint32_t)W.g_h + (p % tp) / (uint32_t)W.g_w);
        const uint32_t pix = (uint32_t)y * (uint32_t)imgw + (uint32_t)x;
        // this pixel's samples in the wave, in sample order
        uint32_t s = (uint32_t)(W.base / ((uint64_t)W.g_s * W.npix)) * (uint32_t)W.g_s;
        float4 acc = film[pix];
        bool any = false;
        for (;; ++s) {
            const uint64_t g = tile2_index(W, p, s);
            if (g >= end) break;
            if (g < W.base) continue;
            const float4 r = P.rad[g - W.base];
            acc.x += smax(0.f, r.x);
            acc.y += smax(0.f, r.y);
            acc.z += smax(0.f, r.z);
            any = true;
        }
        if (any) film[pix] = acc;
        return;
    }
    if (W.tiled == 3) {
        ragged_pixel(p, (uint32_t)imgw, (uint32_t)(W.npix / imgw), x, y);
        const uint64_t first = (uint64_t)p * (uint64_t)W.spp, past = first + (uint64_t)W.spp;
        uint64_t g = first < W.base ? W.base : first;
        const uint64_t stop = past < end ? past : end;
        if (g >= stop) return;
        const uint32_t pix = (uint32_t)y * (uint32_t)imgw + (uint32_t)x;
        float4 acc = film[pix];
        for (; g < stop; ++g) {
            const float4 r = P.rad[g - W.base];
            acc.x += smax(0.f, r.x);
            acc.y += smax(0.f, r.y);
            acc.z += smax(0.f, r.z);
        }
        film[pix] = acc;
        return;
    }
    frame_pixel(p, imgw, W.tiled, x, y);
    const uint32_t pix = (uint32_t)y * (uint32_t)imgw + (uint32_t)x;
    uint64_t s_first = W.base / (uint64_t)W.npix;
    uint64_t g = s_first * (uint64_t)W.npix + p;
    if (g < W.base) g += (uint64_t)W.npix;
    if (g >= end) return;
    float4 acc = film[pix];
    for (; g < end; g += (uint64_t)W.npix) {
        float4 r = P.rad[g - W.base];
        acc.x += smax(0.f, r.x);
        acc.y += smax(0.f, r.y);
        acc.z += smax(0.f, r.z);
    }
    film[pix] = acc;
}

// Copies per-sample max(0, L) to out[(pixel * spp + sample) * 3], pixel the
// index in the pixel list, or y * imgw + x for a full frame.
__global__ void k_collect(PathState P, WaveDesc W, float* out, int spp, int imgw) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.count) return;
    uint64_t g = W.base + (uint64_t)i;
    uint64_t srel = g / (uint64_t)W.npix, pidx = g % (uint64_t)W.npix;
    if (!W.pix_xy && W.tiled) {
        int x, y;
        uint32_t s;
        wave_path(W, g, imgw, x, y, s);
        srel = s;
        pidx = (uint64_t)y * (uint64_t)imgw + (uint64_t)x;
    }
    float4 r = P.rad[i];
    float* o = out + (pidx * (uint64_t)spp + srel) * 3;
    o[0] = smax(0.f, r.x); o[1] = smax(0.f, r.y); o[2] = smax(0.f, r.z);
}

// Mean, gamma and 8-bit conversion (rendererptls.cpp:175-180).
__global__ void k_finish(const float4* film, int npix, float inv_spp, float* hdr, uint8_t* rgb8) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float4 a = film[p];
    float m[3] = {a.x * inv_spp, a.y * inv_spp, a.z * inv_spp};
    for (int k = 0; k < 3; ++k) {
        if (hdr) hdr[3 * p + k] = m[k];
        if (rgb8) {
            float g = powf(m[k], (float)(1.0 / 2.2)) * 255.0f;
            g = smin(255.0f, smax(0.0f, g));
            rgb8[3 * p + k] = (uint8_t)(int)g;
        }
    }
}

// ---------------------------------------------------------------- online cache
// Adds the cache prediction of each query: L += T * max(0, nrc(x)).
__global__ void k_nrc_apply(PathState P, NrcCtx C, const float* __restrict__ pred) {
    const int n = (int)C.counters[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int slot = C.q_slot[i];
        float4 t = C.q_thr[i], r = P.rad[slot];
        const float* o = pred + 3 * (size_t)i;
        P.rad[slot] = make_float4(r.x + t.x * fmaxf(0.f, o[0]), r.y + t.y * fmaxf(0.f, o[1]), r.z + t.z * fmaxf(0.f, o[2]), 0.f);
    }
}

// Training targets: radiance the path gathered from the vertex on, divided by
// the throughput that reached the vertex; channels with negligible
// throughput copy the luminance-weighted value, and targets are clamped.
__global__ void k_nrc_targets(PathState P, NrcCtx C, float* __restrict__ y, float clamp_max) {
    const int n = min((int)C.counters[1], C.tcap);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int slot = C.t_slot[i];
        float4 a = P.rad[slot], b = C.t_before[i], t = C.t_thr[i];
        float d[3] = {a.x - b.x, a.y - b.y, a.z - b.z}, tt[3] = {t.x, t.y, t.z};
        float tsum = tt[0] + tt[1] + tt[2], dsum = d[0] + d[1] + d[2];
        for (int k = 0; k < 3; ++k) {
            float v = tt[k] > 1e-4f ? d[k] / tt[k] : (tsum > 1e-4f ? dsum / tsum : 0.f);
            if (!(v >= 0.f)) v = 0.f;  // NaN or negative
            y[3 * (size_t)i + k] = fminf(v, clamp_max);
        }
    }
}

// ---------------------------------------------------------------- single queries
// One ray per lane, `take` rays per warp. MINB: minimum resident blocks per
// SM; WIDE: the four-wide walk.
template <int MINB, bool WIDE>
__global__ void __launch_bounds__(128, MINB) k_intersect(DeviceScene S, int n, int take, const float* __restrict__ o,
                                                         const float* __restrict__ d, int* __restrict__ tri,
                                                         float* __restrict__ t, float* __restrict__ b1,
                                                         float* __restrict__ b2, uint32_t* err) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * take + lane;
    if (lane >= take || i >= n) return;
    float tt, u, v;
    const int k = query_hit<WIDE>(S, mk(o[3 * i], o[3 * i + 1], o[3 * i + 2]), mk(d[3 * i], d[3 * i + 1], d[3 * i + 2]), tt, u, v, err);
    tri[i] = k >= 0 ? __float_as_int(__ldg(&S.tri_geo[3 * k]).w) : -1;
    t[i] = tt; b1[i] = u; b2[i] = v;
}

// The emitters' radiance from their materials (the light table's layout,
// upload_scene).
__global__ void k_set_emission(float4* __restrict__ lights, const int32_t* __restrict__ light_mat,
                               const nr_material* __restrict__ mats, int num_lights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_lights) return;
    const nr_material& M = mats[light_mat[i]];
    for (int k = 0; k < 3; ++k) lights[6 * (size_t)i + k].w = M.c0[k];
}

struct ListRng {
    const float* u;
    int i;
    __device__ float next() { return i < 4 ? u[i++] : 0.5f; }
};

__global__ void k_material_probe(DeviceScene S, int mat, int n, const float* wo, const float* nrm, const float* wi,
                                 const float* uv, const float* u, float* f, float* pdf, float* wi_s) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f3 a = mk(wo[3 * i], wo[3 * i + 1], wo[3 * i + 2]), nn = mk(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]);
    f3 b = mk(wi[3 * i], wi[3 * i + 1], wi[3 * i + 2]);
    MatView M = load_mat(S, mat, mk(uv[3 * i], uv[3 * i + 1], uv[3 * i + 2]));
    f3 ff = mat_bxdf(M, a, nn, b);
    pdf[i] = mat_pdf(M, a, nn, b);
    ListRng r{u + 4 * i, 0};
    f3 ws = mat_sample(M, r, a, nn);
    f[3 * i] = ff.x; f[3 * i + 1] = ff.y; f[3 * i + 2] = ff.z;
    wi_s[3 * i] = ws.x; wi_s[3 * i + 1] = ws.y; wi_s[3 * i + 2] = ws.z;
}

// ---------------------------------------------------------------- launchers
static int g_trace_blocks = 0, g_shadow_blocks = 0, g_num_sms = 1;

void launch_setup(int num_sms) {
    g_num_sms = num_sms > 0 ? num_sms : 1;
    int b1 = 0, b2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_trace<false, 1>, 128, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, k_shadow<false, true>, 128, 0);
    g_trace_blocks = num_sms * (b1 > 0 ? b1 : 1);
    g_shadow_blocks = num_sms * (b2 > 0 ? b2 : 1);
}

void launch_raygen(const PathState& P, const WaveDesc& W, const nr_camera& cam, float film_h, const Policy& pol,
                   cudaStream_t st) {
    k_raygen<<<(W.count + 255) / 256, 256, 0, st>>>(P, W, cam, film_h, pol);
}

static int count_grid(int cap);

void launch_bounce(const PathState& P, const DeviceScene& S, const Policy& pol, int capacity, int max_count,
                   cudaStream_t st, cudaEvent_t* ev, bool count, const NrcCtx* nrc) {
    const bool sorted = P.sort.place[0] != nullptr;
    if (ev) cudaEventRecord(ev[0], st);
    switch ((count ? 4 : 0) + (pol.trav ? 1 + P.sort.input : 3 * P.sort.input)) {
        case 0: k_trace<false, 0><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 1: k_trace<false, 1><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 2: k_trace<false, 2><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 3: k_trace<false, 3><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 4: k_trace<true, 0><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 5: k_trace<true, 1><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        case 6: k_trace<true, 2><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
        default: k_trace<true, 3><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity); break;
    }
    if (P.sort.bucket_after) k_bucket<<<std::max(1, std::min((max_count + 1023) / 1024, g_num_sms * 32)), 256, 0, st>>>(P, S, capacity);
    if (ev) cudaEventRecord(ev[1], st);
    // the shading kernels stride over their device counts; max_count (an
    // upper bound of their sum) and NR_SHADE_ROUNDS size the grids
    int shade_blocks = (max_count + 127) / 128;
    if (shade_blocks < 1) shade_blocks = 1;
    const int most = g_num_sms * NR_SHADE_MINB * NR_SHADE_ROUNDS;
    if (shade_blocks > most) shade_blocks = most;
    PathState Q = P;
    if (sorted) {  // shading appends the continuing paths beside, the sort moves them into queue_out
        Q.queue_out = P.sort.queue;
        for (int k = 0; k < 2; ++k) cudaMemsetAsync(P.sort.hist[k], 0, (size_t)P.sort.buckets() * 4, st);
    }
    if (nrc) launch_shade<true>(Q, S, pol, capacity, capacity, shade_blocks, *nrc, st);
    else launch_shade<false>(Q, S, pol, capacity, max_count, shade_blocks, NrcCtx{}, st);
    if (sorted) {
        k_ray_scan<<<dim3(P.sort.buckets() / 4096u, 2), 1024, 0, st>>>(P.sort);
        k_ray_scan_parts<<<2, 1024, 0, st>>>(P.sort);
        k_ray_order<<<dim3(g_num_sms * ORDER_BLOCKS, 2), 256, 0, st>>>(P);
    }
    if (ev) cudaEventRecord(ev[2], st);
    float4* tb = (nrc && nrc->direct) ? nrc->t_before : nullptr;
    switch ((count ? 2 : 0) + pol.trav) {
        case 0: k_shadow<false, false><<<g_shadow_blocks, 128, 0, st>>>(P, S, tb); break;
        case 1: k_shadow<false, true><<<g_shadow_blocks, 128, 0, st>>>(P, S, tb); break;
        case 2: k_shadow<true, false><<<g_shadow_blocks, 128, 0, st>>>(P, S, tb); break;
        default: k_shadow<true, true><<<g_shadow_blocks, 128, 0, st>>>(P, S, tb); break;
    }
    if (pol.envis) k_env_fold<<<count_grid(P.sh_cap), 256, 0, st>>>(P, tb);
    if (ev) cudaEventRecord(ev[3], st);
    k_advance<<<1, 1, 0, st>>>(P.counters);
}

void launch_tail(const PathState& P, const DeviceScene& S, const Policy& pol, int capacity, const NrcCtx* nrc,
                 cudaStream_t st) {
    // the four-wide walk up to the count where it stops paying
    const int walk = pol.trav == 0 ? 1 : (S.wide && capacity <= 300000 ? 3 : 2);
    const uint32_t sms = (uint32_t)g_num_sms;
    // one round of resident blocks, fewer where there is not a path for each warp
    const int blocks = std::min(g_num_sms * (walk == 3 ? NR_TAIL_MINB_WIDE : NR_TAIL_MINB), (capacity + 3) / 4);
    const NrcCtx C = nrc ? *nrc : NrcCtx{};
    switch (walk + (nrc ? 3 : 0)) {
        case 1: k_tail<false, 1><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
        case 2: k_tail<false, 2><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
        case 3: k_tail<false, 3><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
        case 4: k_tail<true, 1><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
        case 5: k_tail<true, 2><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
        default: k_tail<true, 3><<<blocks, 128, 0, st>>>(P, S, pol, C, sms); break;
    }
}

void launch_trace(const PathState& P, const DeviceScene& S, const Policy& pol, int capacity, cudaStream_t st) {
    if (pol.trav) k_trace<false, 2><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity);
    else k_trace<false, 3><<<g_trace_blocks, 128, 0, st>>>(P, S, capacity);
}
void launch_advance(uint32_t* counters, cudaStream_t st) { k_advance<<<1, 1, 0, st>>>(counters); }
int shadow_grid() { return g_shadow_blocks; }

void launch_reset_counters(uint32_t* counters, cudaStream_t st) { k_reset_counters<<<1, 32, 0, st>>>(counters); }

// The counts live on the device: grid-stride loops over a grid sized for
// the capacity, at most eight 256-thread blocks per SM.
static int count_grid(int cap) {
    int b = (cap + 255) / 256;
    const int most = 8 * g_num_sms;
    return b < 1 ? 1 : (b > most ? most : b);
}
void launch_sort_recorded(const PathState& P, const DeviceScene& S, int capacity, cudaStream_t st) {
    k_sort_recorded<<<count_grid(capacity), 256, 0, st>>>(P, S, capacity);
}
void launch_nrc_apply(const PathState& P, const NrcCtx& C, const float* pred, int cap, cudaStream_t st) {
    k_nrc_apply<<<count_grid(cap), 256, 0, st>>>(P, C, pred);
}
void launch_nrc_targets(const PathState& P, const NrcCtx& C, float* y, float clamp_max, cudaStream_t st) {
    k_nrc_targets<<<count_grid(C.tcap), 256, 0, st>>>(P, C, y, clamp_max);
}

void launch_film(const PathState& P, const WaveDesc& W, float4* film, int imgw, cudaStream_t st) {
    k_film<<<(W.npix + 255) / 256, 256, 0, st>>>(P, W, film, imgw);
}

void launch_collect(const PathState& P, const WaveDesc& W, float* out, int spp, int imgw, cudaStream_t st) {
    k_collect<<<(W.count + 255) / 256, 256, 0, st>>>(P, W, out, spp, imgw);
}

void launch_finish(const float4* film, int npix, float inv_spp, float* hdr, uint8_t* rgb8, cudaStream_t st) {
    k_finish<<<(npix + 255) / 256, 256, 0, st>>>(film, npix, inv_spp, hdr, rgb8);
}

// A call of few rays lasts as long as its slowest warp, and a warp as long as
// its slowest ray in every phase: the rays are spread over the warps the chip
// holds (32 per SM), one round of them up to 156k rays, and take the four-wide
// walk. Many rays want warps in flight more than registers or short walks. us
// a call, 200k triangles, 4096 / 65,536 / 262,144 camera rays: 154 / 170 / 205
// with closest_hit and full warps, 85 / 125 / 172 with closest_hit_query
// spread, 71 / 108 / 140 four-wide; 1M triangles, 2 M rays off its surfaces in
// no order: 1387 with closest_hit, 1063 / 1012 / 970 with closest_hit_query at
// 8 / 10 / 12 blocks per SM. Measured and dropped: those rays sorted by origin
// and direction first, 923, but 1100 against 271 where a million camera rays
// came in order already.
void launch_intersect(const DeviceScene& S, int n, const float* o, const float* d, int* tri, float* t, float* b1,
                      float* b2, uint32_t* err, cudaStream_t st) {
    const int64_t warps = (int64_t)g_num_sms * 32;
    const int take = (int)std::max<int64_t>(1, std::min<int64_t>(32, (n + warps - 1) / warps));
    const unsigned blocks = (unsigned)(((int64_t)n + 4 * take - 1) / (4 * take));
    if (n < (1 << 19) && S.wide) k_intersect<8, true><<<blocks, 128, 0, st>>>(S, n, take, o, d, tri, t, b1, b2, err);
    else k_intersect<12, false><<<blocks, 128, 0, st>>>(S, n, take, o, d, tri, t, b1, b2, err);
}

void launch_set_emission(float4* lights, const int32_t* light_mat, const nr_material* mats, int num_lights, cudaStream_t st) {
    if (num_lights > 0) k_set_emission<<<(num_lights + 127) / 128, 128, 0, st>>>(lights, light_mat, mats, num_lights);
}

void launch_material_probe(const DeviceScene& S, int mat, int n, const float* wo, const float* nrm, const float* wi,
                           const float* uv, const float* u, float* f, float* pdf, float* wi_s, cudaStream_t st) {
    k_material_probe<<<(n + 127) / 128, 128, 0, st>>>(S, mat, n, wo, nrm, wi, uv, u, f, pdf, wi_s);
}

}  // namespace nr
