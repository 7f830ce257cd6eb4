// cov_map.cuh -- the kernels of the transform engine's maps (cov_lns.cu), one
// instantiation per number of layers and alphabet size, compiled by
// cov_map_low.cu (up to 5 layers) and cov_map_high.cu (more).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "cov_map_plan.h"

#define LNS_MAXR 8
#define MAP_LOW_NT 256
#define MAP_HIGH_NT 384

struct MapGeom {
    int q, n, R;
    uint32_t T, Tp;                 // words and columns of a low tile
    int32_t *out;                   // the map, or
    uint16_t *cnt16;                // the counts (saturated)
};

typedef void (*MapLow)(MapGeom, int, int, uint32_t, const uint64_t *, const uint64_t *, const int32_t *, uint32_t,
                       uint32_t, int32_t *, int);
typedef void (*MapHigh)(MapGeom, int, int, int, uint32_t, uint32_t, const int32_t *, int32_t *, int);

// the kernels for at most that many layers and the alphabet size q
void map_kernels_3(int q, MapLow *low, MapHigh *high);
void map_kernels_5(int q, MapLow *low, MapHigh *high);
void map_kernels_7(int q, MapLow *low, MapHigh *high);
void map_kernels_9(int q, MapLow *low, MapHigh *high);

#ifdef COV_MAP_KERNELS

// ----------------------------------------------------------- the maps -----
// A map is C_R[x] = #{marked y : d(x,y) <= R} by cumulative layers: with j of
// the n axes done, C_d[x] counts the marked y that agree with x on the other
// axes and lie within d of it on these.  Taking an axis more, along a line
// with sums T_d = sum of C_d,
//     C_d[x] += T_{d-1} - C_{d-1}[x].
// Two facts keep the layers few.  With j axes done C_d = C_j for d > j, so
// layers 0..min(R, j) are held and an axis adds one (C_{j+1} = T_j).  With k
// axes left only layers R-k..R can reach C_R, so below that they are dropped.
//
// The first nb axes come from the masks: C_d of a block of q^nb words is a
// population count of its mask and the words within d.

// A tile's element e holds its layers side by side, layer d at e * RC + d: RC
// is odd, so the lanes of a warp fall in 32 banks, and the layers of an
// element are constant offsets from one address.
//
// One axis over `nfib` lines of q elements at element stride st: NL layers
// from Ls on, the lowest left as it is, a new one added above the highest when
// GROW.  Each thread owns whole lines.  With the alphabet size Q known at
// compile time a line's Q x NL counts are read once into registers; Q = 0 is
// the form for any q.
template <int NT, int RC, int NL, bool GROW, int Q>
__device__ __forceinline__ void map_axis(int32_t *Ls, int q, uint32_t nfib, uint32_t st)
{
    // f / st by a float reciprocal: f < 2^24, so the estimate is off by at
    // most one and one correction makes it exact
    const float rinv = 1.0f / (float)st;
    for (uint32_t f = threadIdx.x; f < nfib; f += NT) {
        int o = (int)((float)f * rinv);
        int i = (int)f - o * (int)st;
        if (i < 0) { o--; i += (int)st; } else if (i >= (int)st) { o++; i -= (int)st; }
        int32_t *const p = Ls + ((uint32_t)o * st * (uint32_t)q + (uint32_t)i) * RC;
        const uint32_t sp = st * RC;
        constexpr int NS = GROW ? NL : NL - 1;            // line sums needed
        int32_t S[NS > 0 ? NS : 1];
        if constexpr (Q > 0) {
            int32_t v[Q][NL];
#pragma unroll
            for (int a = 0; a < Q; a++)
#pragma unroll
                for (int d = 0; d < NL; d++) v[a][d] = p[(uint32_t)a * sp + d];
#pragma unroll
            for (int d = 0; d < NS; d++) {
                S[d] = 0;
#pragma unroll
                for (int a = 0; a < Q; a++) S[d] += v[a][d];
            }
#pragma unroll
            for (int a = 0; a < Q; a++) {
#pragma unroll
                for (int d = 1; d < NL; d++) p[(uint32_t)a * sp + d] = v[a][d] + S[d - 1] - v[a][d - 1];
                if constexpr (GROW) p[(uint32_t)a * sp + NL] = S[NL - 1];
            }
        } else {
#pragma unroll
            for (int d = 0; d < NS; d++) S[d] = 0;
            for (int a = 0; a < q; a++) {
#pragma unroll
                for (int d = 0; d < NS; d++) S[d] += p[(uint32_t)a * sp + d];
            }
            for (int a = 0; a < q; a++) {
                int32_t *const pe = p + (uint32_t)a * sp;
                int32_t below = pe[0];
#pragma unroll
                for (int d = 1; d < NL; d++) {
                    const int32_t old = pe[d];
                    pe[d] = old + S[d - 1] - below;
                    below = old;
                }
                if constexpr (GROW) pe[NL] = S[NL - 1];
            }
        }
    }
}

// nl layers (at most RC) from Ls on
template <int NT, int RC, int Q>
__device__ __forceinline__ void map_axis_n(int nl, bool grow, int32_t *Ls, int q, uint32_t nfib, uint32_t st)
{
    switch (nl) {
#define MAP_AXIS_CASE(K) \
    case K: \
        if constexpr (K <= RC) { \
            if (!grow) { map_axis<NT, RC, K, false, Q>(Ls, q, nfib, st); break; } \
            if constexpr (K < RC) map_axis<NT, RC, K, true, Q>(Ls, q, nfib, st); \
        } \
        break;
    MAP_AXIS_CASE(1) MAP_AXIS_CASE(2) MAP_AXIS_CASE(3) MAP_AXIS_CASE(4) MAP_AXIS_CASE(5) MAP_AXIS_CASE(6)
    MAP_AXIS_CASE(7) MAP_AXIS_CASE(8) MAP_AXIS_CASE(9)
#undef MAP_AXIS_CASE
    }
}

// Between two sweeps the layers of a word lie side by side, as in the reading
// sweep's shared memory: layer lo + i of column c at (c * slots + i), so that
// a row of a strip is one run of 16-byte copies straight into its tile.  For
// their alignment a tile of T = q^k words takes Tp columns, T rounded up to a
// multiple of four; the columns in between hold anything.

__device__ __forceinline__ void map_put(const MapGeom &g, uint32_t x, int32_t s)
{
    if (g.out) g.out[x] = s;
    else g.cnt16[x] = (uint16_t)min(s, 65535);
}

// Axes 0..k-1 on contiguous tiles of T = q^k words, `ntile` of them from tile0
// on, to columns from `to` on.  The first nb axes come from the masks um
// (lowball: the words of a block within d of each); with A0 instead (word
// counts of a code), from its values.
template <int RC, int Q>
static __global__ void __launch_bounds__(MAP_LOW_NT) k_map_low(MapGeom g, int k, int nb, uint32_t blk,
                                                        const uint64_t *__restrict__ um,
                                                        const uint64_t *__restrict__ lowball,
                                                        const int32_t *__restrict__ A0, uint32_t tile0, uint32_t ntile,
                                                        int32_t *to, int slots)
{
    extern __shared__ __align__(16) int32_t Ls[];
    const int q = Q > 0 ? Q : g.q;
    const uint32_t T = g.T;
    uint64_t *const tab = reinterpret_cast<uint64_t *>(Ls + g.Tp * RC);
    uint64_t *const ms = tab + blk * (uint32_t)(nb + 1);
    const int lo = map_lo(g.n, g.R, k), hi = map_hi(g.R, k);
    if (um) for (uint32_t i = threadIdx.x; i < blk * (uint32_t)(nb + 1); i += MAP_LOW_NT) tab[i] = lowball[i];
    for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
        const uint32_t x0 = (tile0 + t) * T;
        int done = 0;
        if (um) {
            const uint32_t b0 = x0 / blk;
            for (uint32_t i = threadIdx.x; i < T / blk; i += MAP_LOW_NT) ms[i] = __ldg(&um[b0 + i]);
            __syncthreads();
            done = nb;
            const int h0 = map_hi(g.R, nb);
            for (uint32_t e = threadIdx.x; e < T; e += MAP_LOW_NT) {
                const uint32_t z = e / blk, y = e - z * blk;
                const uint64_t m = ms[z];
                Ls[e * RC] = (int32_t)((m >> y) & 1u);
                for (int d = 1; d <= h0; d++)
                    Ls[e * RC + (uint32_t)d] = __popcll(m & tab[y * (uint32_t)(nb + 1) + (uint32_t)d]);
            }
        } else {
            __syncthreads();
            for (uint32_t e = threadIdx.x; e < T; e += MAP_LOW_NT) Ls[e * RC] = A0[x0 + e];
        }
        __syncthreads();
        uint32_t st = 1;
        for (int j = 0; j < done; j++) st *= (uint32_t)q;
        for (; done < k; done++, st *= (uint32_t)q) {
            const int l0 = map_lo(g.n, g.R, done), h0 = map_hi(g.R, done);
            map_axis_n<MAP_LOW_NT, RC, Q>(h0 - l0 + 1, map_hi(g.R, done + 1) > h0, Ls + l0, q, T / (uint32_t)q, st);
            __syncthreads();
        }
        if (k == g.n) {
            for (uint32_t e = threadIdx.x; e < T; e += MAP_LOW_NT) map_put(g, x0 + e, Ls[e * RC + (uint32_t)g.R]);
        } else if (slots == RC && lo == 0) {
            const int4 *src = reinterpret_cast<const int4 *>(Ls);
            int4 *dst = reinterpret_cast<int4 *>(to + (size_t)t * g.Tp * RC);
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < g.Tp * RC / 4; i += MAP_LOW_NT) dst[i] = src[i];
        } else {
            int32_t *dst = to + (size_t)t * g.Tp * (uint32_t)slots;
            for (uint32_t e = threadIdx.x; e < T; e += MAP_LOW_NT)
                for (int d = lo; d <= hi; d++) dst[e * (uint32_t)slots + (uint32_t)(d - lo)] = Ls[e * RC + (uint32_t)d];
        }
        // the next tile's masks land beside the layers, its layers after a barrier
    }
}

// Axes j0..j0+gsz-1 on strips: q^gsz rows of W = 2^lw consecutive columns, row
// r of a strip s columns after row r - 1; `ntile` strips.  Column c of `from`
// is column c of `to`, or, after the last axis, word (c / Tp) * T + c % Tp.
template <int RC, int Q>
static __global__ void __launch_bounds__(MAP_HIGH_NT, RC <= 5 ? 2 : 1) k_map_high(MapGeom g, int j0, int gsz, int lw, uint32_t s,
                                                                           uint32_t ntile, const int32_t *from,
                                                                           int32_t *to, int slots)
{
    extern __shared__ __align__(16) int32_t Ls[];
    const int q = Q > 0 ? Q : g.q;
    const uint32_t W = 1u << lw;
    uint32_t rows = 1;
    for (int j = 0; j < gsz; j++) rows *= (uint32_t)q;
    const uint32_t E = rows << lw, nstrip = (s + W - 1) >> lw;
    const int end = j0 + gsz;
    const int li = map_lo(g.n, g.R, j0);
    const int lo = map_lo(g.n, g.R, end), hi = map_hi(g.R, end);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(Ls);
    const uint32_t run = (RC << lw) / 4;              // 16-byte pieces of a whole row
    for (uint32_t t = blockIdx.x; t < ntile; t += gridDim.x) {
        const uint32_t o = t / nstrip, c0 = (t - o * nstrip) << lw;
        const uint32_t w = min(W, s - c0);            // columns of the strip, a multiple of four
        const size_t base = (size_t)o * rows * s + c0;
        __syncthreads();
        // every piece is in flight at once, with no registers
        for (uint32_t i = threadIdx.x; i < rows * run; i += MAP_HIGH_NT) {
            const uint32_t r = i / run, p = i - r * run;
            if (p < w * RC / 4)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + 16u * i),
                             "l"(from + (base + (size_t)r * s) * RC + 4 * p) : "memory");
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        uint32_t st = W;
        for (int done = j0; done < end; done++, st *= (uint32_t)q) {
            const int l0 = map_lo(g.n, g.R, done), h0 = map_hi(g.R, done);
            map_axis_n<MAP_HIGH_NT, RC, Q>(h0 - l0 + 1, map_hi(g.R, done + 1) > h0, Ls + (l0 - li), q, E / (uint32_t)q, st);
            __syncthreads();
        }
        if (end == g.n) {
            const int32_t *res = Ls + (g.R - li);
            // a thread's column is the same in every row (W divides the CTA)
            const uint32_t c = threadIdx.x & (W - 1), z = (c0 + c) / g.Tp, y = c0 + c - z * g.Tp;
            const uint32_t sw = s / g.Tp * g.T;       // words between two rows
            if (c < w && y < g.T) {
                const uint32_t x = (uint32_t)o * rows * sw + z * g.T + y;
#pragma unroll 4
                for (uint32_t r = threadIdx.x >> lw; r < rows; r += MAP_HIGH_NT >> lw)
                    map_put(g, x + r * sw, res[((r << lw) + c) * RC]);
            }
        } else {
            const uint32_t nl = (uint32_t)(hi - lo + 1);
            for (uint32_t e = threadIdx.x; e < E; e += MAP_HIGH_NT) {
                const uint32_t r = e >> lw, c = e & (W - 1);
                if (c >= w) continue;
                int32_t *dst = to + (base + (size_t)r * s + c) * (uint32_t)slots;
                const int32_t *src = Ls + e * RC + (uint32_t)(lo - li);
#pragma unroll
                for (uint32_t d = 0; d < RC; d++)
                    if (d < nl) dst[d] = src[d];
            }
        }
    }
}

// alphabet sizes with their own kernels (others run the Q = 0 form)
#define MAP_Q_LIST(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

template <int RC>
static void map_kernels_rc(int q, MapLow *low, MapHigh *high)
{
    switch (q) {
#define MAP_CASE_Q(QQ) case QQ: *low = k_map_low<RC, QQ>; *high = k_map_high<RC, QQ>; break;
    MAP_Q_LIST(MAP_CASE_Q)
#undef MAP_CASE_Q
    default: *low = k_map_low<RC, 0>; *high = k_map_high<RC, 0>; break;
    }
}

#endif
