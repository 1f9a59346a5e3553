// am_device.cuh -- device helpers shared by the engine's kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "am_internal.h"

namespace am {

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    using type = float4;
};
template <>
struct Vec4<double> {
    using type = double4;
};
template <typename T>
using vec4_t = typename Vec4<T>::type;

template <typename T>
__device__ __forceinline__ vec4_t<T> ld4(const T *p)
{
    return *reinterpret_cast<const vec4_t<T> *>(p);
}
template <typename T>
__device__ __forceinline__ void st4(T *p, vec4_t<T> v)
{
    *reinterpret_cast<vec4_t<T> *>(p) = v;
}

// ---------------------------------------------------------------- keys
__device__ __forceinline__ int key_bit(const uint32_t *key, int k) { return (key[k >> 5] >> (k & 31)) & 1; }

// 64-bit mix (splitmix64 finaliser)
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Hash of a packed key = sum over words of mix64(word, position).  Additive,
// so flipping one bit updates it in O(1).
__host__ __device__ __forceinline__ uint64_t word_term(uint32_t w, int pos)
{
    return mix64(((uint64_t)(uint32_t)pos << 32) | (uint64_t)w);
}

__device__ __forceinline__ uint64_t flip_hash(uint64_t h, uint32_t word, int k)
{
    const int pos = k >> 5;
    return h - word_term(word, pos) + word_term(word ^ (1u << (k & 31)), pos);
}

// slot value: [fingerprint 32][tag 1][id 31]; tag 1 = candidate of the
// current wave, 0 = committed region
__device__ __forceinline__ uint32_t fp_of(uint64_t h) { return (uint32_t)(h >> 32); }
__device__ __forceinline__ unsigned long long slot_value(uint32_t fp, int cand, uint32_t id)
{
    return ((unsigned long long)fp << 32) | ((unsigned long long)(cand ? 1u : 0u) << 31) | (id & 0x7fffffffu);
}

// ---------------------------------------------------------------- tiles of a wave
// The composition's tiles of R regions, the classes (ChunkDev) one after the
// other from the longest (class 1) to the shortest, so that the CTAs' rounds
// hold tiles of about the same length.  Every second round runs backwards over
// the CTAs: the CTA with the longest tile of one round gets the shortest of the
// next.
struct WavePlan {
    int cnt[kMaxLayers];        // regions per class
    int tile0[kMaxLayers + 1];  // first tile of each class
    int R, layers;
};

__device__ __forceinline__ int plan_class_tiles(const WavePlan &w, int c, int R) { return (w.cnt[c] + R - 1) / R; }
__device__ __forceinline__ int plan_tiles(const WavePlan &w, int R)
{
    int n = 0;
    for (int c = 0; c < w.layers; ++c) n += plan_class_tiles(w, c, R);
    return n;
}
// (one warp) The wave's plan, and its R: the first of R0, R0 + step, ... whose tiles
// fit `slots`, at most rmax (at most 32 steps away); R0 is a slot's share of the
// regions.  The classes' counts, the sizes and the tiles are a lane's each (one
// thread's loops over them took 1 to 2 us of every wave on GB300).
__device__ __forceinline__ int plan_wave(WavePlan &w, const ChunkDev &ch, int layers, int count, int slots, int rmax, int step)
{
    const int lane = threadIdx.x & 31;
    const int n = ch.order ? layers : 1;
    if (lane == 0) w.layers = n;
    if (lane < n) w.cnt[lane] = ch.order ? ch.ccount[lane] : count;
    __syncwarp();
    const int per = (count + slots - 1) / slots, r0 = min(rmax, max((per + step - 1) / step, 1) * step);
    const int mine = r0 + step * lane;
    const bool fits = mine >= rmax || plan_tiles(w, mine) <= slots;
    const int R = min(rmax, r0 + step * (__ffs(__ballot_sync(0xffffffffu, fits)) - 1));
    int sum = lane < n ? plan_class_tiles(w, lane, R) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += below;
    }
    if (lane == 0) {
        w.R = R;
        w.tile0[0] = 0;
    }
    if (lane < n) w.tile0[lane + 1] = sum;
    return R;
}
// the tile of round j on CTA b of G, -1 when there is none
__device__ __forceinline__ int plan_tile(const WavePlan &w, int j, int b, int G)
{
    const long long t = (long long)j * G + ((j & 1) ? G - 1 - b : b);
    return t < w.tile0[w.layers] ? (int)t : -1;
}
__device__ __forceinline__ int plan_rounds(const WavePlan &w, int G) { return (w.tile0[w.layers] + G - 1) / G; }
__device__ __forceinline__ int plan_class(const WavePlan &w, int t)
{
    int c = 0;
    while (t >= w.tile0[c + 1]) ++c;
    return c + 1;
}

// wave position of region r of tile t, class c
__device__ __forceinline__ int tile_pos(const WavePlan &w, const ChunkDev &ch, int t, int c, int r)
{
    const int idx = (t - w.tile0[c - 1]) * w.R + r;
    return ch.order ? ch.order[(size_t)(c - 1) * ch.order_cap + idx] : idx;
}
// One region of a tile: x its own rows' slot, y its parent's, z the plane it
// was entered through (its row changes sign between the two; -1 for class 1),
// w its wave position.
__device__ __forceinline__ int4 tile_region(const WavePlan &w, const RegionsDev &reg, const ChunkDev &ch, long long head,
                                            int t, int c, int r)
{
    const int rl = tile_pos(w, ch, t, c, r);
    int4 o;
    o.x = (int)row_slot(ch, head, rl);
    o.y = o.x;
    o.z = -1;
    o.w = rl;
    if (c > 1) {
        o.y = (int)ring_slot(ch, reg.parent[head + rl]);
        o.z = reg.start[head + rl];
    }
    return o;
}
__device__ __forceinline__ int tile_nreg(const WavePlan &w, int t, int c)
{
    return min(w.R, w.cnt[c - 1] - (t - w.tile0[c - 1]) * w.R);
}
// a region's constraint row: the rows before jend from its parent's slot
// (rewritten by no region of this wave), the plane it was entered through with
// the other sign; the rest from its own
template <typename T>
__device__ __forceinline__ vec4_t<T> tile_row(const T *cons, size_t rstride, const int4 &ri, int row, int jend)
{
    vec4_t<T> v = ld4<T>(cons + (size_t)(uint32_t)(row < jend ? ri.y : ri.x) * rstride + (size_t)row * 4);
    if (row == ri.z) {
        v.x = -v.x;
        v.y = -v.y;
        v.z = -v.z;
        v.w = -v.w;
    }
    return v;
}

// ---------------------------------------------------------------- 3x3
// Cramer's rule for A x + b = 0 with rows (r0, r1, r2) -- the reference's
// solve_3x3 (backend/inc/kernel.h:553-571).  Returns the determinant.
template <typename S>
__device__ __forceinline__ S det3(S a0, S a1, S a2, S a3, S a4, S a5, S a6, S a7, S a8)
{
    return a0 * (a4 * a8 - a5 * a7) - a1 * (a3 * a8 - a5 * a6) + a2 * (a3 * a7 - a4 * a6);
}

template <typename S>
__device__ __forceinline__ S solve3(const S *r0, const S *r1, const S *r2, S *x)
{
    const S d0 = det3<S>(r0[0], r0[1], r0[2], r1[0], r1[1], r1[2], r2[0], r2[1], r2[2]);
    const S d1 = det3<S>(-r0[3], r0[1], r0[2], -r1[3], r1[1], r1[2], -r2[3], r2[1], r2[2]);
    const S d2 = det3<S>(r0[0], -r0[3], r0[2], r1[0], -r1[3], r1[2], r2[0], -r2[3], r2[2]);
    const S d3 = det3<S>(r0[0], r0[1], -r0[3], r1[0], r1[1], -r1[3], r2[0], r2[1], -r2[3]);
    x[0] = d1 / d0;
    x[1] = d2 / d0;
    x[2] = d3 / d0;
    return d0;
}

// get_i_j (backend/inc/kernel.h:607-622): pair index x -> (i, j), i > j,
// along anti-diagonals of i + j, clamped to ij_max - 1.
__device__ __forceinline__ void get_i_j(int x, int ij_max, int &i, int &j)
{
    const int k = x / 2;
    const int a = (int)ceilf(sqrtf(2 * k + 2.25f) - 1.5f);
    const int r = x - a * (a + 1);
    const int A = 2 * a + r / (a + 1);
    const int B = r % (a + 1);
    i = (A + 1) / 2 + B + 1;
    j = A + 1 - i;
    i = i < ij_max ? i : ij_max - 1;
    j = j < ij_max ? j : ij_max - 1;
}

} // namespace am
