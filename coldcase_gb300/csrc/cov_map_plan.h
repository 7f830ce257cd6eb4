// cov_map_plan.h -- how the sweeps of the transform engine's maps
// (cov_map.cuh, cov_lns.cu) group the axes of a cell, and what memory they
// take; and the bound on the steps of its greedy.  Host arithmetic only, so
// that it compiles without CUDA.
#pragma once
#include <cstddef>
#include <cstdint>
#include <algorithm>

#ifdef __CUDACC__
#define MAP_HD __host__ __device__ __forceinline__
#else
#define MAP_HD static inline
#endif

#define MAP_MAXN 16                 // most axes
#define MAP_SMEM_MAX (200 * 1024)   // shared memory of one map tile (bytes)
#define MAP_SMEM_LOW (84 * 1024)    // of a low tile: two CTAs an SM at least
#define MAP_SMEM_HIGH (112 * 1024)  // of a strip: two
#define MAP_W_MIN 8                 // narrowest strip
#define MAP_L2_BYTES (80 << 20)     // layers of the parts that are in flight between two sweeps

// layers of a tile with `done` of the n axes done: map_lo .. map_hi
MAP_HD int map_lo(int n, int R, int done) { return R - (n - done) > 0 ? R - (n - done) : 0; }
MAP_HD int map_hi(int R, int done) { return done < R ? done : R; }

static inline long long map_ipow(long long q, int k)
{
    long long p = 1;
    while (k-- > 0) p *= q;
    return p;
}

// a sweep of `layers` layers: kernels for 3, 5, 7 and 9, so that the registers
// and the shared memory of an element stay few where the layers are
static inline int map_slots(int layers) { return layers <= 3 ? 3 : layers <= 5 ? 5 : layers <= 7 ? 7 : 9; }

// layers that a strip sweep of axes j0 .. j0+gsz-1 holds of an element
static inline int map_strip_slots(int n, int R, int j0, int gsz)
{
    return map_slots(map_hi(R, j0 + gsz) - map_lo(n, R, j0) + 1);
}

static inline uint32_t map_cols(int q, int k) { return ((uint32_t)map_ipow(q, k) + 3u) & ~3u; }

// a low tile at `slots` layers an element: the layers, the table of the
// blocks' balls, the masks
static inline size_t map_low_smem(int q, int slots, int k, int nb, uint32_t blk)
{
    return (size_t)map_cols(q, k) * slots * 4 + (size_t)blk * (nb + 1) * 8 + (size_t)map_ipow(q, k) / blk * 8;
}

struct MapPlan {
    int kl = 0, ng = 0, gs[MAP_MAXN] = {}, slots[MAP_MAXN] = {};   // low axes, strip groups: their axes and layers
    uint32_t parts = 1, at_once = 1;
    size_t scratch_ints = 0, whole_ints = 0;
    // The word counts that a transform may start from instead of the masks lie
    // at the end of the memory of the layers that reach the last sweep (two
    // groups or more: what a part writes there ends before the counts of the
    // parts after it), else in words of their own behind the scratch.
    size_t counts_at = 0;               // in the layers' memory, or behind scratch_ints
    size_t counts_ints = 0;             // words of their own

    // the low kernel works at the slots of its reader where they hold its layers
    int low_slots(int R) const { return std::max(map_slots(map_hi(R, kl) + 1), ng ? slots[0] : 0); }
};

// How the axes of N = q^n words are grouped (blocks of blk = q^nb words are
// the masks'): the low ones in tiles at two CTAs an SM or more, the others in
// strips of at least eight columns at two, in as few groups as that allows,
// the larger ones first.
static inline void map_plan(MapPlan &p, int q, int n, int R, uint32_t N, int nb, uint32_t blk)
{
    p = MapPlan{};
    p.kl = nb;
    while (p.kl < n && map_low_smem(q, map_slots(map_hi(R, p.kl + 1) + 1), p.kl + 1, nb, blk) <= MAP_SMEM_LOW) p.kl++;
    const int m = n - p.kl;
    p.counts_ints = N;
    if (m == 0) return;                  // one tile holds the space: no strips, nothing between sweeps
    int gmax = 1;
    while (gmax < m && map_ipow(q, gmax + 1) * MAP_W_MIN * map_slots(R + 1) * 4 <= MAP_SMEM_HIGH) gmax++;
    p.ng = (m + gmax - 1) / gmax;
    for (int i = 0, left = m; i < p.ng; i++) {
        p.gs[i] = (left + p.ng - i - 1) / (p.ng - i);
        left -= p.gs[i];
    }
    for (int i = 0, j0 = p.kl; i < p.ng; j0 += p.gs[i++]) p.slots[i] = map_strip_slots(n, R, j0, p.gs[i]);
    // All groups but the last work within the words that share the last
    // group's digits.  A few such parts at a time go through them, so that
    // what a sweep writes is still in L2 when the next one reads it.
    p.parts = p.ng >= 2 ? (uint32_t)map_ipow(q, p.gs[p.ng - 1]) : 1u;
    int most = 0;
    for (int i = 0; i < std::max(1, p.ng - 1); i++) most = std::max(most, p.slots[i]);
    const long long cols = (long long)(N / p.parts) / map_ipow(q, p.kl) * map_cols(q, p.kl);
    p.at_once = (uint32_t)std::max(1LL, std::min<long long>(p.parts, MAP_L2_BYTES / (cols * most * 4)));
    p.scratch_ints = (size_t)cols * p.at_once * most;
    if (p.ng < 2) return;
    p.whole_ints = (size_t)cols * p.parts * p.slots[p.ng - 1];
    p.counts_ints = 0;
    p.counts_at = p.whole_ints - N;
}

// Most steps of a greedy launch that places up to `room` words and leaves for
// a fresh map after eval_cap exact counts without a placement: a step that
// places none counts one candidate at least, so eval_cap of them come before
// a placement or the end.  (The kernel gives up beyond it.)
static inline long long greedy_max_steps(int room, int eval_cap) { return ((long long)room + 1) * (eval_cap + 1LL); }
