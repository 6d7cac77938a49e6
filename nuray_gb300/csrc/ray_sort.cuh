// Counting sort of a bounce's new rays by where they start and where they go,
// so that the 32 rays of a warp walk much of the same tree: shading leaves
// them in the order of the pixels they come from, which says little about
// either after the first vertex, and nothing about the directions before.
//
// Key: the Morton code of the origin's cell (cubic cells over the scene box)
// above the direction's cell on an octahedral map. Shading gives every ray its
// place in its bucket with one atomic as it appends it (ray_place); a scan
// turns the bucket sizes into offsets, and a pass over the queue writes each
// ray's entry to offset + place. The order within a bucket is whatever the
// atomics made it: nothing depends on it, each path's sums have one writer.
#pragma once
#include "nr_device.cuh"

namespace nr {

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // bit i of the low 10 to bit 3 i
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}
// x as a cell of [0, 2^bits - 1]; NaN gives 0
__device__ __forceinline__ uint32_t ray_cell(float x, int bits) {
    return (uint32_t)fminf(fmaxf(x, 0.f), (float)((1 << bits) - 1));
}
__device__ __forceinline__ uint32_t ray_key(const DeviceScene& S, const RaySort& s, f3 o, f3 d) {
    const float k = s.cells_per_unit;
    const uint32_t m = spread3(ray_cell((o.x - S.root_lo[0]) * k, s.origin_bits)) |
                       (spread3(ray_cell((o.y - S.root_lo[1]) * k, s.origin_bits)) << 1) |
                       (spread3(ray_cell((o.z - S.root_lo[2]) * k, s.origin_bits)) << 2);
    const float l = __fdividef(1.0f, fabsf(d.x) + fabsf(d.y) + fabsf(d.z));
    float u = d.x * l, v = d.z * l;
    if (d.y < 0.f) {
        const float a = copysignf(1.f - fabsf(v), u);
        v = copysignf(1.f - fabsf(u), v);
        u = a;
    }
    const float h = 0.5f * (float)(1 << s.dir_bits);
    uint32_t du = ray_cell(u * h + h, s.dir_bits);
    const uint32_t dv = ray_cell(v * h + h, s.dir_bits);
    if (dv & 1u) du = ((1u << s.dir_bits) - 1u) - du;  // every other row backwards: neighbours in the code are neighbours
    return (((m << s.dir_bits) | dv) << s.dir_bits) | du;
}
// The place of a ray appended as entry q.
__device__ __forceinline__ void ray_place(const DeviceScene& S, const RaySort& s, int which, uint32_t q, f3 o, f3 d) {
    const uint32_t k = ray_key(S, s, o, d);
    s.place[which][q] = make_uint2(k, atomicAdd(&s.hist[which][k], 1u));
}

// Exclusive sum over the 1024 threads of a block; total: the block's sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t own, uint32_t* sums, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31u) sums[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32u) {
        const uint32_t a = sums[lane];
        uint32_t b = a;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= (uint32_t)o) b += y;
        }
        sums[lane] = b - a;
        if (lane == 31u) sums[32] = b;
    }
    __syncthreads();
    total = sums[32];
    return x - own + sums[threadIdx.x >> 5];
}

// Offsets of 4096 buckets within their block; the block's total in part.
__global__ void __launch_bounds__(1024) k_ray_scan(RaySort s) {
    __shared__ uint32_t sums[33];
    uint4* p = reinterpret_cast<uint4*>(s.hist[blockIdx.y] + (size_t)blockIdx.x * 4096) + threadIdx.x;
    const uint4 v = *p;
    uint32_t total;
    const uint32_t e = block_scan(v.x + v.y + v.z + v.w, sums, total);
    *p = make_uint4(e, e + v.x, e + v.x + v.y, e + v.x + v.y + v.z);
    if (threadIdx.x == 0) s.part[blockIdx.y][blockIdx.x] = total;
}
// The blocks' own offsets, one block for each of the two sorts.
__global__ void __launch_bounds__(1024) k_ray_scan_parts(RaySort s) {
    __shared__ uint32_t sums[33];
    uint32_t* part = s.part[blockIdx.x];
    const uint32_t parts = s.buckets() / 4096u;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < parts; base += 1024u) {
        const uint32_t i = base + threadIdx.x;
        uint32_t total;
        const uint32_t e = block_scan(i < parts ? part[i] : 0u, sums, total);
        if (i < parts) part[i] = carry + e;
        carry += total;
        __syncthreads();
    }
}
// Where the entry placed at (bucket, place) = a belongs.
__device__ __forceinline__ uint32_t ray_offset(const RaySort& s, int which, uint2 a) {
    return s.hist[which][a.x] + s.part[which][a.x >> 12] + a.y;
}

}  // namespace nr
