// cov_verify.cu -- GB300 (sm_103a) verification kernels for covering codes.
//
//   * exact per-word minimum distance to a code (the distance transform),
//     computed as axis passes of the line-min recurrence
//         D'(x) = min(D(x), 1 + min_a D(x with x_j := a)).
//     After the passes over axes 0..n-1, D(x) is the
//     Hamming distance from x to the nearest codeword -- the `best` array of
//     cov/verify_independent.py:144-186 -- and #{x : D(x) > R} is the
//     uncovered count that cov/verify_cov.py:109-230 returns.
//     Few codewords: every tile of the word space is made from the code
//     alone, with the values of a line or of a block of two digits as masks,
//     and each distance is written once.  Many: uint8 values, the low axes
//     of a contiguous tile, then the high axes of column strips, each group
//     worked in shared memory.  The histogram of D is folded into the last
//     pass.
//   * coverage multiplicity cnt[x] = #{i : d(x,c_i) <= R} by marking every
//     codeword's ball (covsearch2e.c:353-380, 958-967) tile by tile in shared
//     memory (cov_tiles.cuh).
#include <cmath>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <vector>
#include <algorithm>
#include "cov_common.cuh"
#include "cov_tiles.cuh"
#include "../../include/covgpu.h"

#define DT_TILE_MAX   65536    // bytes of the contiguous low-axes tile (several CTAs per SM)
#define DT_TILE_BIG   (200 * 1024)  // a tile of one CTA per SM, used when it saves a sweep
#define DT_NT_BIG     1024     // threads of a big-tile CTA
#define DT_STRIP_MAX  98304    // bytes of a high-axes strip
#define DT_STRIP_W    32       // narrowest strip (columns); strips widen while they fit
#define DT_NT         512

#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { \
    fprintf(stderr, "covgpu: CUDA error %s at %s:%d\n", cudaGetErrorString(e_), __FILE__, __LINE__); \
    return -(100 + (int)e_); } } while (0)

struct DtGeom {
    int q, n;
    uint32_t N;
    uint32_t pw[COV_MAXN + 1];   // pw[k] = q^k
    int inf;                     // n + 1
};

// --------------------------------------------------------- code bitmap ----
// Index of the word with the n digits c, all ones (which is no index) when a
// digit lies outside the alphabet: the sum alone could be another word's, or
// lie past the end of the scratch that it indexes.
__device__ __forceinline__ uint32_t dt_word(const uint8_t *__restrict__ c, int n, uint32_t q)
{
    uint32_t x = 0;
    bool word = true;
    for (int j = 0; j < n; j++) {
        const uint32_t a = c[j];
        word = word && a < q;
        x = x * q + a;
    }
    return word ? x : 0xffffffffu;
}

__global__ void k_dt_bitmap(const uint8_t *__restrict__ code, int M, DtGeom g, uint32_t *bm)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const uint32_t x = dt_word(code + (size_t)i * g.n, g.n, (uint32_t)g.q);
        if (x != 0xffffffffu) atomicOr(&bm[x >> 5], 1u << (x & 31));
    }
}

// histogram update aggregated over the lanes holding the same value
__device__ __forceinline__ void dt_hist_add(int *sh, int v)
{
    const unsigned act = __activemask();
    const unsigned same = __match_any_sync(act, v);
    if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&sh[v], __popc(same));
}

// One line-min pass over packed bytes: `nfib` fibres of Q 32-bit words, word
// a of fibre f at  base(f) + a*stride  (a < Q), base(f) = (f / inner) *
// Q*stride + (f % inner).  Each word holds 4 independent lines (one per
// byte).  The bytes are worked as two pairs of 16-bit lanes (bytes 0,2 and
// 1,3), where the minimum of three values and min(m + 1, n + 1) are single
// dynamic-programming instructions (__vimin3_u16x2, __viaddmin_u16x2).
template <int Q>
__device__ __forceinline__ void dt_pass4(uint32_t *w, int nfib, int stride, int inner, uint32_t inf4)
{
    const uint32_t inf2 = inf4 & 0x00ff00ffu;
    // f / inner by a float reciprocal: f < 2^24, so the estimate is off by
    // at most one and one correction makes it exact
    const float rinv = 1.0f / (float)inner;
    for (int f = threadIdx.x; f < nfib; f += blockDim.x) {
        int o = (int)((float)f * rinv);
        int i = f - o * inner;
        if (i < 0) { o--; i += inner; } else if (i >= inner) { o++; i -= inner; }
        uint32_t *b = w + o * Q * stride + i;
        uint32_t e[Q], d[Q];                     // bytes 0,2 and bytes 1,3 of each word
#pragma unroll
        for (int a = 0; a < Q; a++) {
            const uint32_t x = b[a * stride];
            e[a] = __byte_perm(x, 0u, 0x4240);
            d[a] = __byte_perm(x, 0u, 0x4341);
        }
        uint32_t me = e[0], md = d[0];
#pragma unroll
        for (int a = 1; a + 1 < Q; a += 2) {
            me = __vimin3_u16x2(me, e[a], e[a + 1]);
            md = __vimin3_u16x2(md, d[a], d[a + 1]);
        }
        if ((Q & 1) == 0) {
            me = __vminu2(me, e[Q - 1]);
            md = __vminu2(md, d[Q - 1]);
        }
        const uint32_t ce = __viaddmin_u16x2(me, 0x00010001u, inf2);
        const uint32_t cd = __viaddmin_u16x2(md, 0x00010001u, inf2);
#pragma unroll
        for (int a = 0; a < Q; a++)
            b[a * stride] = __byte_perm(__vminu2(e[a], ce), __vminu2(d[a], cd), 0x6240);
    }
}

// Pass 1: tiles of T = Q^k contiguous words (the low k axes), from the code
// bitmap.  In shared memory a tile is T/Q rows -- the Q words of one line of
// the lowest axis -- each padded to 4*ceil(Q/4) bytes, so that every axis
// above the lowest moves whole 32-bit words.  The lowest axis is taken while
// loading: a word is 0 on the code, 1 if its line holds a codeword, else
// n+1.  When k == n this is the whole transform and the histogram is taken
// here.
template <int Q>
__global__ void __launch_bounds__(DT_NT_BIG)
k_dt_low(DtGeom g, int k, const uint32_t *__restrict__ bm, uint8_t *__restrict__ D,
         unsigned long long *hist)
{
    extern __shared__ __align__(16) uint32_t dt_w[];
    __shared__ int sh[COV_MAXN + 2];
    constexpr int WPR = (Q + 3) >> 2;            // 32-bit words per row
    constexpr uint32_t RB = 4u * WPR;            // padded row bytes
    uint32_t T = 1;
    for (int j = 0; j < k; j++) T *= (uint32_t)Q;
    const int rows = (int)(T / (uint32_t)Q);
    const uint32_t inf = (uint32_t)g.inf, inf4 = inf * 0x01010101u;
    const uint32_t ntile = g.N / T;
    const bool last = (k == g.n) && hist != nullptr;
    uint8_t *dt_b = reinterpret_cast<uint8_t *>(dt_w);
    if (threadIdx.x < COV_MAXN + 2) sh[threadIdx.x] = 0;
    for (uint32_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const uint32_t x0 = tile * T;
        __syncthreads();
        for (int r = threadIdx.x; r < rows; r += blockDim.x) {
            const uint32_t xr = x0 + (uint32_t)r * (uint32_t)Q;
            // Q bits of the row from at most two bitmap words
            const uint32_t lo = __ldg(&bm[xr >> 5]);
            const uint32_t hi = ((xr & 31) + (uint32_t)Q > 32) ? __ldg(&bm[(xr >> 5) + 1]) : 0u;
            const uint32_t bits = (uint32_t)(((((uint64_t)hi << 32) | lo) >> (xr & 31)) & ((1ull << Q) - 1));
            const uint32_t fill = bits ? 1u : inf;
#pragma unroll
            for (int w = 0; w < WPR; w++) {
                uint32_t v = 0;
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const int a = 4 * w + b;
                    const uint32_t byte = a >= Q ? inf : (((bits >> a) & 1u) ? 0u : fill);
                    v |= byte << (8 * b);
                }
                dt_w[r * WPR + w] = v;
            }
        }
        __syncthreads();
        int inner = WPR;                       // rows of axis j: stride Q^(j-1) rows
        for (int j = 1; j < k; j++, inner *= Q) {
            dt_pass4<Q>(dt_w, rows / Q * WPR, inner, inner, inf4);
            __syncthreads();
        }
        // out: the tile is T contiguous bytes of D; the 4-byte-aligned
        // interior goes out as whole words (byte b of the tile is row b / Q,
        // column b % Q of the padded rows), the unaligned ends as bytes
        const uint32_t head = min((4u - (uint32_t)(reinterpret_cast<uintptr_t>(D + x0) & 3u)) & 3u, T);
        const uint32_t nw = (T - head) >> 2;
        for (uint32_t e = threadIdx.x; e < head + ((T - head) & 3u); e += blockDim.x) {
            const uint32_t b = e < head ? e : head + 4 * nw + (e - head);
            const uint32_t r = b / (uint32_t)Q;
            const uint8_t v = dt_b[r * RB + (b - r * (uint32_t)Q)];
            D[x0 + b] = v;
            if (last) dt_hist_add(sh, v);
        }
        for (uint32_t wi = threadIdx.x; wi < nw; wi += blockDim.x) {
            const uint32_t b0 = head + 4 * wi;
            uint32_t r = b0 / (uint32_t)Q, a = b0 - r * (uint32_t)Q, v = 0;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t byte = dt_b[r * RB + a];
                v |= byte << (8 * t);
                if (last) dt_hist_add(sh, (int)byte);
                if (++a == (uint32_t)Q) { a = 0; r++; }
            }
            *reinterpret_cast<uint32_t *>(D + x0 + b0) = v;
        }
    }
    __syncthreads();
    if (last && threadIdx.x < g.n + 2 && sh[threadIdx.x])
        atomicAdd(&hist[threadIdx.x], (unsigned long long)sh[threadIdx.x]);
}

// the aligned 32-bit word that holds byte p
__device__ __forceinline__ uint32_t *dt_word_of(uint8_t *p)
{
    return reinterpret_cast<uint32_t *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
}

// Pass 2+: the axes of group [j0, j0+gsz) (in-word strides Q^j0 .. ), for a
// strip of W = 32 << lw consecutive positions below the group: rows of W
// bytes, W/4 words, so each pass moves whole words.  W is as wide as the
// shared memory allows for the group's Q^gsz rows, so that a group of few
// rows (the last axes of a long word) still moves long contiguous runs.
// A row starts at any byte (the strides are powers of Q), so it is moved
// as 32-bit words: each loaded word is two aligned words funnel-shifted by
// the row's misalignment (the second only when it holds bytes of the row),
// and each row goes out as aligned words plus at most three bytes at either
// end.  Every word touched holds a byte of the row, so no access leaves it.
template <int Q>
__global__ void __launch_bounds__(DT_NT)
k_dt_high(DtGeom g, int j0, int gsz, int lw, int last_, uint8_t *__restrict__ D, unsigned long long *hist)
{
    const bool last = last_ && hist != nullptr;
    extern __shared__ __align__(16) uint32_t dt_w[];
    __shared__ int sh[COV_MAXN + 2];
    const int lwb = lw + 5;                      // log2 of the strip width in bytes
    const int lww = lwb - 2;                     // log2 of the words per row
    const uint32_t W = 1u << lwb;
    const uint32_t WW = W >> 2;
    uint8_t *dt_b = reinterpret_cast<uint8_t *>(dt_w);
    const uint32_t inf4 = (uint32_t)g.inf * 0x01010101u;
    uint32_t s = 1;                              // stride of the lowest axis in the group
    for (int j = 0; j < j0; j++) s *= (uint32_t)Q;
    uint32_t rows = 1;
    for (int j = 0; j < gsz; j++) rows *= (uint32_t)Q;
    const uint32_t span = rows * s;              // words spanned by one value of the outer digits
    const uint32_t outer = g.N / span;
    const uint32_t nstrip = (s + W - 1) >> lwb;
    const unsigned long long ntiles = (unsigned long long)outer * nstrip;
    if (threadIdx.x < COV_MAXN + 2) sh[threadIdx.x] = 0;
    const uint32_t totw = rows << lww;
    for (unsigned long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint32_t o = (uint32_t)(tile / nstrip);
        const uint32_t c0 = (uint32_t)(tile - (unsigned long long)o * nstrip) << lwb;
        const uint32_t w = min(W, s - c0);       // bytes of each row in this strip
        uint8_t *const Db = D + (size_t)o * span + c0;
        __syncthreads();
        // word k of row r: bytes 4k..4k+3 of the row at Db + r*s (n+1
        // past w); eight words of a thread in flight before their stores
        for (uint32_t e0 = threadIdx.x; e0 < totw; e0 += 8 * blockDim.x) {
            uint32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t e = e0 + (uint32_t)u * blockDim.x;
                const uint32_t r = e >> lww, c = (e & (WW - 1)) << 2;
                v[u] = inf4;
                if (e < totw && c < w) {
                    uint8_t *p = Db + (size_t)r * s + c;
                    const uint32_t m = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
                    const uint32_t need = min(4u, w - c);
                    const uint32_t *pa = dt_word_of(p);
                    const uint32_t lo = pa[0];
                    const uint32_t hi = m + need > 4u ? pa[1] : 0u;
                    uint32_t x = __funnelshift_r(lo, hi, 8u * m);
                    if (need < 4u) {
                        const uint32_t keep = (1u << (8u * need)) - 1u;
                        x = (x & keep) | (inf4 & ~keep);
                    }
                    v[u] = x;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t e = e0 + (uint32_t)u * blockDim.x;
                if (e < totw) dt_w[e] = v[u];
            }
        }
        __syncthreads();
        int inner = (int)WW;                     // row stride Q^j
        for (int j = 0; j < gsz; j++, inner *= Q) {
            dt_pass4<Q>(dt_w, (int)(rows / (uint32_t)Q) * (int)WW, inner, inner, inf4);
            __syncthreads();
        }
        // out: row r's aligned words from its first 4-byte boundary on, then
        // the ends (at most 3 bytes each) by the thread of the row's last word
        for (uint32_t e = threadIdx.x; e < totw; e += blockDim.x) {
            const uint32_t r = e >> lww, k = e & (WW - 1);
            uint8_t *p0 = Db + (size_t)r * s;
            const uint32_t head = min((4u - (uint32_t)(reinterpret_cast<uintptr_t>(p0) & 3u)) & 3u, w);
            const uint32_t nwr = (w - head) >> 2;
            if (k < nwr) {
                const uint32_t lo = dt_w[(r << lww) + k];
                const uint32_t hi = head ? dt_w[(r << lww) + k + 1] : 0u;
                const uint32_t x = __funnelshift_r(lo, hi, 8u * head);
                *reinterpret_cast<uint32_t *>(p0 + head + 4 * k) = x;
                if (last) {
#pragma unroll
                    for (int b = 0; b < 4; b++) dt_hist_add(sh, (int)((x >> (8 * b)) & 0xffu));
                }
            }
            if (k == WW - 1) {
                const uint8_t *row = dt_b + ((size_t)r << lwb);
                for (uint32_t b = 0; b < head; b++) {
                    p0[b] = row[b];
                    if (last) atomicAdd(&sh[row[b]], 1);
                }
                for (uint32_t b = head + 4 * nwr; b < w; b++) {
                    p0[b] = row[b];
                    if (last) atomicAdd(&sh[row[b]], 1);
                }
            }
        }
    }
    __syncthreads();
    if (last && threadIdx.x < g.n + 2 && sh[threadIdx.x])
        atomicAdd(&hist[threadIdx.x], (unsigned long long)sh[threadIdx.x]);
}

// ------------------------------------------- the transform of few codewords --
// When the code is small beside a tile of T = q^nl words (the low nl digits),
// a tile needs no other tile: every codeword enters it at its low digits with
// the distance of its high digits to the tile's as the starting value, and
// the nl low axes finish the transform.  One launch writes each distance
// once; nothing is read but the code.
//
// A line of the lowest axis is one 32-bit word, (m << 16) | mask: D = m at
// the positions in mask and m + 1 elsewhere.  That is exact because distances
// along an axis already taken differ by at most one (D is 1-Lipschitz in it),
// and it stays true through the other axes.  With E the minimum over the q
// lines of a fibre -- the least m, and the union of the masks that have it --
// a line becomes min(line, E + 1): itself if its m is E's, the union of both
// masks if it is one more, E + 1 otherwise.  A line element therefore costs
// about 11 instructions a pass for q words, where a byte of its own costs
// about two a word (and q bytes of shared memory instead of four).
// Bound by instruction issue (72 % of the slots at 8^9, 19 lane-instructions
// a word; DRAM 14 % busy): 8^10 with 2549 codewords takes 0.68 ms, against
// 4.5 ms for a tile pass and two strip sweeps of bytes.  q = 5..8 mostly take
// the blocks below.
#define DT_TILES_NT 512
#define DT_TILES_KEEP 8          // codewords a thread keeps between the two marking passes
#define DT_TILES_SMEM (100 * 1024)

// shared-memory slot of line l: for q = 8 the three low digits of l are
// folded into the bank bits, so that a warp's fibres of the first three axes
// fall in 32 banks (unswizzled: 8-way and 4-way conflicts).  XOR-linear.
template <int Q>
__device__ __forceinline__ uint32_t dt_slot(uint32_t l)
{
    if constexpr (Q == 8) return l ^ ((l >> 3) & 7u) ^ (((l >> 6) & 3u) << 3);
    return l;
}

// per codeword: {nibbles of the high digits, (line of the low digits' tile << 4) | position}
template <int Q>
__global__ void k_dt_records(const uint8_t *__restrict__ code, int M, DtGeom g, int nl, uint2 *__restrict__ rec)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const uint32_t x = dt_word(code + (size_t)i * g.n, g.n, (uint32_t)Q);
        uint32_t hi = x / g.pw[nl], h = 0;
        const uint32_t lo = x - hi * g.pw[nl];
        for (int j = 0; j < g.n - nl; j++) { h |= (hi % (uint32_t)Q) << (4 * j); hi /= (uint32_t)Q; }
        rec[i] = x == 0xffffffffu ? make_uint2(0u, 0xffffffffu)
                                  : make_uint2(h, (dt_slot<Q>(lo / (uint32_t)Q) << 4) | (lo % (uint32_t)Q));
    }
}

__device__ __forceinline__ uint32_t dt_nibble_dist(uint32_t a, uint32_t b)
{
    uint32_t x = a ^ b;
    x |= x >> 1;
    x |= x >> 2;
    return (uint32_t)__popc(x & 0x11111111u);
}

// four distances from four mask bits: m where a bit is set, m + 1 elsewhere;
// m1 holds m + 1 in every byte
__device__ __forceinline__ uint32_t dt_expand4(uint32_t bits, uint32_t m1)
{
    return m1 - ((bits * 0x00204081u) & 0x01010101u);
}

template <int Q>
__global__ void __launch_bounds__(DT_TILES_NT, Q <= 10 ? 3 : 1)
k_dt_tiles(DtGeom g, int nl, const uint2 *__restrict__ rec, int M, uint8_t *__restrict__ D, unsigned long long *hist)
{
    extern __shared__ __align__(16) uint32_t dt_w[];
    __shared__ int sh[COV_MAXN + 2];
    constexpr uint32_t FULL = (1u << Q) - 1u;
    const uint32_t T = g.pw[nl], lines = g.pw[nl - 1], ntile = g.N / T;
    const uint32_t nt = blockDim.x;
    const int nh = g.n - nl;
    if (threadIdx.x < COV_MAXN + 2) sh[threadIdx.x] = 0;
    for (uint32_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        uint32_t hp = 0;
        {
            uint32_t t = tile;
            for (int j = 0; j < nh; j++) { hp |= (t % (uint32_t)Q) << (4 * j); t /= (uint32_t)Q; }
        }
        __syncthreads();
        for (uint32_t l = threadIdx.x; l < lines; l += nt) dt_w[l] = ((uint32_t)g.inf << 16) | FULL;
        __syncthreads();
        // least starting value of every line, then the positions that have it
        // kept: (starting value << 28) | (line << 4) | position, all ones for none
        uint32_t kept[DT_TILES_KEEP];
        const bool keep = (uint32_t)M <= nt * DT_TILES_KEEP;
        if (keep) {
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++) {
                const uint32_t i = threadIdx.x + (uint32_t)u * nt;
                kept[u] = 0xffffffffu;
                if ((uint32_t)u * nt < (uint32_t)M && i < (uint32_t)M) {
                    const uint2 r = __ldg(&rec[i]);
                    if (r.y != 0xffffffffu) kept[u] = (dt_nibble_dist(r.x, hp) << 28) | r.y;
                }
            }
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++)
                if ((uint32_t)u * nt < (uint32_t)M && kept[u] != 0xffffffffu) atomicMin(&dt_w[(kept[u] & 0x0fffffffu) >> 4], (kept[u] >> 28) << 16);
        } else {
            for (uint32_t i = threadIdx.x; i < (uint32_t)M; i += nt) {
                const uint2 r = __ldg(&rec[i]);
                if (r.y != 0xffffffffu) atomicMin(&dt_w[r.y >> 4], dt_nibble_dist(r.x, hp) << 16);
            }
        }
        __syncthreads();
        if (keep) {
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++) {
                if ((uint32_t)u * nt >= (uint32_t)M || kept[u] == 0xffffffffu) continue;
                const uint32_t at = (kept[u] & 0x0fffffffu) >> 4;
                if ((dt_w[at] >> 16) == kept[u] >> 28) atomicOr(&dt_w[at], 1u << (kept[u] & 15u));
            }
        } else {
            for (uint32_t i = threadIdx.x; i < (uint32_t)M; i += nt) {
                const uint2 r = __ldg(&rec[i]);
                if (r.y != 0xffffffffu && (dt_w[r.y >> 4] >> 16) == dt_nibble_dist(r.x, hp))
                    atomicOr(&dt_w[r.y >> 4], 1u << (r.y & 15u));
            }
        }
        __syncthreads();
        // the other low axes, a fibre of Q lines at a time
        uint32_t inner = 1;
        for (int j = 1; j < nl; j++, inner *= (uint32_t)Q) {
            const float rinv = 1.0f / (float)inner;   // f < 2^24: one correction makes f / inner exact
            const uint32_t p1 = dt_slot<Q>(inner), p2 = dt_slot<Q>(2u * inner), p4 = dt_slot<Q>(4u * inner);
            for (uint32_t f = threadIdx.x; f < lines / (uint32_t)Q; f += nt) {
                int o = (int)((float)f * rinv);
                int i = (int)f - o * (int)inner;
                if (i < 0) { o--; i += (int)inner; } else if (i >= (int)inner) { o++; i -= (int)inner; }
                const uint32_t b = dt_slot<Q>((uint32_t)o * (uint32_t)Q * inner + (uint32_t)i);
                uint32_t v[Q], ad[Q];
#pragma unroll
                for (int a = 0; a < Q; a++) {
                    if constexpr (Q == 8)
                        ad[a] = b ^ ((a & 1) ? p1 : 0u) ^ ((a & 2) ? p2 : 0u) ^ ((a & 4) ? p4 : 0u);
                    else
                        ad[a] = b + (uint32_t)a * inner;
                    v[a] = dt_w[ad[a]];
                }
                uint32_t e = v[0];
#pragma unroll
                for (int a = 1; a < Q; a++) e = min(e, v[a]);
                const uint32_t t0 = (e & 0xffff0000u) + 0x10000u, t1 = t0 + 0x10000u;   // m of E + 1, and one more
                uint32_t w = t0;
#pragma unroll
                for (int a = 0; a < Q; a++)
                    if (v[a] < t0) w |= v[a] & FULL;
#pragma unroll
                for (int a = 0; a < Q; a++)
                    if (v[a] >= t0) dt_w[ad[a]] = v[a] < t1 ? v[a] | w : w;
            }
            __syncthreads();
        }
        if (hist) {
            int m = -1, at = 0, more = 0;             // words at m and at m + 1 of a run of lines
            for (uint32_t l = threadIdx.x; l < lines; l += nt) {
                const uint32_t v = dt_w[l];
                if ((int)(v >> 16) != m) {
                    if (at) atomicAdd(&sh[m], at);
                    if (more) atomicAdd(&sh[m + 1], more);
                    m = (int)(v >> 16);
                    at = more = 0;
                }
                const int c = __popc(v & FULL);
                at += c;
                more += Q - c;
            }
            if (at) atomicAdd(&sh[m], at);
            if (more) atomicAdd(&sh[m + 1], more);
        }
        if (!D) continue;
        uint8_t *const out = D + (size_t)tile * T;
        if (Q == 8 && (reinterpret_cast<uintptr_t>(D) & 7u) == 0) {
            for (uint32_t l = threadIdx.x; l < lines; l += nt) {
                const uint32_t v = dt_w[dt_slot<Q>(l)];
                const uint32_t m1 = ((v >> 16) + 1u) * 0x01010101u;
                reinterpret_cast<uint2 *>(out)[l] = make_uint2(dt_expand4(v & 15u, m1), dt_expand4((v >> 4) & 15u, m1));
            }
            continue;
        }
        // aligned 32-bit words of the tile's T bytes, each from the one, two
        // or (q = 2) three lines that its bytes lie in; the ends as bytes
        const uint32_t head = min((4u - (uint32_t)(reinterpret_cast<uintptr_t>(out) & 3u)) & 3u, T);
        const uint32_t nw = (T - head) >> 2;
        for (uint32_t k = threadIdx.x; k < head + ((T - head) & 3u); k += nt) {
            const uint32_t b = k < head ? k : 4 * nw + k;
            const uint32_t v = dt_w[dt_slot<Q>(b / (uint32_t)Q)];
            out[b] = (uint8_t)((v >> 16) + 1u - ((v >> (b % (uint32_t)Q)) & 1u));
        }
        for (uint32_t k = threadIdx.x; k < nw; k += nt) {
            const uint32_t b = head + 4 * k;
            uint32_t l = b / (uint32_t)Q, a = b - l * (uint32_t)Q;
            uint32_t x = 0, done = 0;
#pragma unroll
            for (int part = 0; part < (Q == 2 ? 3 : 2); part++) {
                if (done < 4u) {
                    const uint32_t v = dt_w[dt_slot<Q>(l)];
                    const uint32_t y = dt_expand4(((v & FULL) >> a) & 15u, ((v >> 16) + 1u) * 0x01010101u);
                    const uint32_t keepm = 0xffffffffu << (8u * done);
                    x = (x & ~keepm) | ((y << (8u * done)) & keepm);
                    done += (uint32_t)Q - a;
                    a = 0;
                    l++;
                }
            }
            *reinterpret_cast<uint32_t *>(out + b) = x;
        }
    }
    __syncthreads();
    if (hist && threadIdx.x < g.n + 2 && sh[threadIdx.x])
        atomicAdd(&hist[threadIdx.x], (unsigned long long)sh[threadIdx.x]);
}

// ------------------------------------------------ the same, block by block --
// For q = 5..8 a block of the two lowest axes, q^2 <= 64 words, is one element:
// its least distance e, the words at e (a0) and the words at e or e + 1 (a1)
// as bit masks; all others are at e + 2, because two words of a block differ
// by two steps at most.  A block starts from the codewords that enter it --
// e is the least starting value, a0 the codewords with it, a1 their rows and
// columns and the codewords one farther -- so that the two lowest axes cost
// nothing; along another axis, with E the least e of a fibre's q blocks and
// U0, U1 the words of the fibre at E and within E + 1, a block becomes
// min(block, E + 1, ...) in a handful of mask operations for q^2 words.
template <int Q> struct DtMask { typedef unsigned long long W; };
template <> struct DtMask<5> { typedef uint32_t W; };
#define DT_BLOCKS_SMEM (100 * 1024)

// bit of word y of a block.  q = 8: the four words of a 32-bit store stand at
// the same bit of the four bytes of a half, so that a shift and a mask make
// four bytes of them.
template <int Q>
__host__ __device__ constexpr int dt_bit(int y)
{
    return Q == 8 ? (y & 3) * 8 + ((y >> 2) & 7) + 32 * (y >> 5) : y;
}

// per codeword: {nibbles of the high digits, (slot of the block << 6) | word}
template <int Q>
__global__ void k_dt_block_records(const uint8_t *__restrict__ code, int M, DtGeom g, int nl, uint2 *__restrict__ rec)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const uint32_t x = dt_word(code + (size_t)i * g.n, g.n, (uint32_t)Q);
        uint32_t hi = x / g.pw[nl], h = 0;
        const uint32_t lo = x - hi * g.pw[nl];
        for (int j = 0; j < g.n - nl; j++) { h |= (hi % (uint32_t)Q) << (4 * j); hi /= (uint32_t)Q; }
        rec[i] = x == 0xffffffffu ? make_uint2(0u, 0xffffffffu)
                                  : make_uint2(h, (dt_slot<Q>(lo / (uint32_t)(Q * Q)) << 6) | (lo % (uint32_t)(Q * Q)));
    }
}

// NT: the most threads of a CTA.  A fibre of q = 6..8 blocks wants the registers
// of 256 threads (8^10 with 2549 codewords 409 -> 370 us, 7^10 with 163 155 ->
// 137); many codewords want the threads (8^9 with 20000: 151 -> 119), and q = 5
// has masks of half the size.
//
// Bound by the integer pipe (65 % at 8^9 with 1000 codewords, 7.2
// lane-instructions a word) and, below some hundred tiles an SM, by the last
// wave.  Against a line an element (k_dt_tiles): 8^10 M 2549 686 -> 370 us (2.9
// TB/s of distances), 7^10 M 163 267 -> 137, 5^12 M 3000 295 -> 169, 6^11 M 300
// 334 -> 230, 7^9 M 1500 57 -> 40.
template <int Q, int NT>
__global__ void __launch_bounds__(NT, NT > 256 ? 2 : 3)
k_dt_blocks(DtGeom g, int nl, const uint2 *__restrict__ rec, int M, uint8_t *__restrict__ D, unsigned long long *hist)
{
    typedef typename DtMask<Q>::W W;
    constexpr uint32_t QQ = Q * Q, HALVES = sizeof(W) / 4;
    constexpr W ALL = (W)(~(W)0) >> (8 * sizeof(W) - QQ);
    struct __align__(2 * sizeof(W)) Planes { W a0, a1; };
    extern __shared__ __align__(16) uint32_t dt_w[];
    __shared__ int sh[COV_MAXN + 4];
    __shared__ W cross[QQ];                        // a word's row and column
    const uint32_t T = g.pw[nl], nblk = T / QQ, ntile = g.N / T;
    Planes *const pl = reinterpret_cast<Planes *>(dt_w);
    uint32_t *const le = dt_w + (size_t)nblk * 2 * HALVES;
    const uint32_t nt = blockDim.x;
    const int nh = g.n - nl;
    if (threadIdx.x < COV_MAXN + 4) sh[threadIdx.x] = 0;
    if (threadIdx.x < QQ) {
        W c = 0;
        const int y = (int)threadIdx.x;
        for (int k = 0; k < Q; k++) c |= ((W)1 << dt_bit<Q>(y / Q * Q + k)) | ((W)1 << dt_bit<Q>(k * Q + y % Q));
        cross[y] = c;
    }
    for (uint32_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        uint32_t hp = 0;
        {
            uint32_t t = tile;
            for (int j = 0; j < nh; j++) { hp |= (t % (uint32_t)Q) << (4 * j); t /= (uint32_t)Q; }
        }
        __syncthreads();
        for (uint32_t l = threadIdx.x; l < nblk; l += nt) le[l] = (uint32_t)g.inf;
        __syncthreads();
        // least starting value of every block, then the masks:
        // (starting value << 28) | (slot << 6) | word, all ones for none
        uint32_t kept[DT_TILES_KEEP];
        const bool keep = (uint32_t)M <= nt * DT_TILES_KEEP;
        auto entry = [&](uint32_t i) {
            const uint2 r = __ldg(&rec[i]);
            return r.y == 0xffffffffu ? r.y : (dt_nibble_dist(r.x, hp) << 28) | r.y;
        };
        auto lower = [&](uint32_t v) {
            if (v != 0xffffffffu) atomicMin(&le[(v & 0x0fffffffu) >> 6], v >> 28);
        };
        auto mark = [&](uint32_t v) {
            if (v == 0xffffffffu) return;
            const uint32_t at = (v & 0x0fffffffu) >> 6, y = v & 63u, e = le[at], s = v >> 28;
            if (s > e + 1u) return;
            uint32_t *const p = dt_w + (size_t)at * 2 * HALVES;
            const W bit = (W)1 << dt_bit<Q>((int)y), c = s == e ? cross[y] : bit;
#pragma unroll
            for (uint32_t h = 0; h < HALVES; h++) {
                const uint32_t b = (uint32_t)(bit >> (16 * h) >> (16 * h)), x = (uint32_t)(c >> (16 * h) >> (16 * h));
                if (s == e && b) atomicOr(&p[h], b);
                if (x) atomicOr(&p[HALVES + h], x);
            }
        };
        if (keep) {
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++) {
                const uint32_t i = threadIdx.x + (uint32_t)u * nt;
                kept[u] = (uint32_t)u * nt < (uint32_t)M && i < (uint32_t)M ? entry(i) : 0xffffffffu;
            }
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++)
                if ((uint32_t)u * nt < (uint32_t)M) lower(kept[u]);
        } else {
            for (uint32_t i = threadIdx.x; i < (uint32_t)M; i += nt) lower(entry(i));
        }
        __syncthreads();
        for (uint32_t l = threadIdx.x; l < nblk; l += nt) {
            const W x = le[l] == (uint32_t)g.inf ? ALL : 0;       // no codeword: every word is at inf
            pl[l].a0 = x;
            pl[l].a1 = x;
        }
        __syncthreads();
        if (keep) {
#pragma unroll
            for (int u = 0; u < DT_TILES_KEEP; u++)
                if ((uint32_t)u * nt < (uint32_t)M) mark(kept[u]);
        } else {
            for (uint32_t i = threadIdx.x; i < (uint32_t)M; i += nt) mark(entry(i));
        }
        __syncthreads();
        // the other low axes, a fibre of Q blocks at a time
        uint32_t inner = 1;
        for (int j = 2; j < nl; j++, inner *= (uint32_t)Q) {
            const float rinv = 1.0f / (float)inner;   // f < 2^24: one correction makes f / inner exact
            const uint32_t p1 = dt_slot<Q>(inner), p2 = dt_slot<Q>(2u * inner), p4 = dt_slot<Q>(4u * inner);
            for (uint32_t f = threadIdx.x; f < nblk / (uint32_t)Q; f += nt) {
                int o = (int)((float)f * rinv);
                int i = (int)f - o * (int)inner;
                if (i < 0) { o--; i += (int)inner; } else if (i >= (int)inner) { o++; i -= (int)inner; }
                const uint32_t b = dt_slot<Q>((uint32_t)o * (uint32_t)Q * inner + (uint32_t)i);
                auto slot = [&](int a) {
                    if constexpr (Q == 8) return b ^ ((a & 1) ? p1 : 0u) ^ ((a & 2) ? p2 : 0u) ^ ((a & 4) ? p4 : 0u);
                    else return b + (uint32_t)a * inner;
                };
                uint32_t e[Q];
                Planes v[Q];
#pragma unroll
                for (int a = 0; a < Q; a++) {
                    e[a] = le[slot(a)];
                    v[a] = pl[slot(a)];
                }
                uint32_t E = e[0];
#pragma unroll
                for (int a = 1; a < Q; a++) E = min(E, e[a]);
                W u0 = 0, u1 = 0;
#pragma unroll
                for (int a = 0; a < Q; a++) {
                    if (e[a] == E) { u0 |= v[a].a0; u1 |= v[a].a1; }
                    if (e[a] == E + 1u) u1 |= v[a].a0;
                }
#pragma unroll
                for (int a = 0; a < Q; a++) {
                    if (e[a] == E) {
                        pl[slot(a)].a1 = v[a].a1 | u0;
                    } else {
                        Planes w{u0, u1};
                        if (e[a] == E + 1u) { w.a0 |= v[a].a0; w.a1 |= v[a].a1; }
                        if (e[a] == E + 2u) w.a1 |= v[a].a0;
                        pl[slot(a)] = w;
                        le[slot(a)] = E + 1u;
                    }
                }
            }
            __syncthreads();
        }
        auto bits = [](W x) {
            if constexpr (sizeof(W) == 8) return __popcll(x);
            else return __popc(x);
        };
        if (hist) {
            int m = -1, at = 0, next = 0, more = 0;    // words at m, m + 1 and m + 2 of a run of blocks
            auto put = [&] {
                if (at) atomicAdd(&sh[m], at);
                if (next) atomicAdd(&sh[m + 1], next);
                if (more) atomicAdd(&sh[m + 2], more);
            };
            for (uint32_t l = threadIdx.x; l < nblk; l += nt) {
                if ((int)le[l] != m) {
                    put();
                    m = (int)le[l];
                    at = next = more = 0;
                }
                const int c0 = bits(pl[l].a0), c1 = bits(pl[l].a1);
                at += c0;
                next += c1 - c0;
                more += (int)QQ - c1;
            }
            put();
        }
        if (!D) continue;
        uint8_t *const out = D + (size_t)tile * T;
        if constexpr (Q == 8) {
            // sixteen words of a block, a quarter of it, a lane (D is 16-byte aligned)
            for (uint32_t x = threadIdx.x; x < nblk * 4u; x += nt) {
                const uint32_t l = dt_slot<Q>(x >> 2), h = (x >> 1) & 1u, sft = (x & 1u) * 4u;
                const uint32_t a0 = dt_w[l * 4u + h] >> sft, a1 = dt_w[l * 4u + 2u + h] >> sft;
                const uint32_t m2 = (le[l] + 2u) * 0x01010101u;
                auto four = [&](int k) { return m2 - ((a0 >> k) & 0x01010101u) - ((a1 >> k) & 0x01010101u); };
                reinterpret_cast<uint4 *>(out)[x] = make_uint4(four(0), four(1), four(2), four(3));
            }
        } else {
            // aligned pieces of 16 bytes, each from the one or two blocks that
            // its bytes lie in; the ends as bytes
            const uint32_t head = min((16u - (uint32_t)(reinterpret_cast<uintptr_t>(out) & 15u)) & 15u, T);
            const uint32_t np = (T - head) >> 4, ends = T - 16u * np;
            for (uint32_t k = threadIdx.x; k < ends; k += nt) {
                const uint32_t x = k < head ? k : 16u * np + k, l = x / QQ, y = x - l * QQ;
                out[x] = (uint8_t)(le[l] + 2u - (uint32_t)((pl[l].a0 >> y) & 1u) - (uint32_t)((pl[l].a1 >> y) & 1u));
            }
            for (uint32_t k = threadIdx.x; k < np; k += nt) {
                const uint32_t x = head + 16u * k, l = x / QQ, y = x - l * QQ;
                const int left = (int)(QQ - y);          // words of block l in the piece
                const Planes v = pl[l];
                uint32_t a0 = (uint32_t)(v.a0 >> y), a1 = (uint32_t)(v.a1 >> y);
                const uint32_t ma = (le[l] + 2u) * 0x01010101u;
                uint32_t mb = ma;
                if (left < 16) {
                    const Planes w = pl[l + 1];
                    a0 |= (uint32_t)w.a0 << left;
                    a1 |= (uint32_t)w.a1 << left;
                    mb = (le[l + 1] + 2u) * 0x01010101u;
                }
                uint32_t r[4];
#pragma unroll
                for (int k4 = 0; k4 < 4; k4++) {
                    const int c = min(max(left - 4 * k4, 0), 4);
                    const uint32_t first = (uint32_t)((1ull << (8 * c)) - 1ull);
                    const uint32_t m2 = (ma & first) | (mb & ~first);
                    r[k4] = m2 - ((((a0 >> (4 * k4)) & 15u) * 0x00204081u) & 0x01010101u) -
                            ((((a1 >> (4 * k4)) & 15u) * 0x00204081u) & 0x01010101u);
                }
                *reinterpret_cast<uint4 *>(out + x) = make_uint4(r[0], r[1], r[2], r[3]);
            }
        }
    }
    __syncthreads();
    if (hist && threadIdx.x < g.n + 2 && sh[threadIdx.x])
        atomicAdd(&hist[threadIdx.x], (unsigned long long)sh[threadIdx.x]);
}

template <int Q>
int dt_blocks_launch(int grid, int nt, size_t smem, cudaStream_t st, const uint8_t *code, int M, const DtGeom &g, int nl,
                     uint2 *rec, uint8_t *D, unsigned long long *hist)
{
    if (M > 0) {
        k_dt_block_records<Q><<<std::min(1024, (M + 255) / 256), 256, 0, st>>>(code, M, g, nl, rec);
        CK(cudaGetLastError());
    }
    if (nt > 256) k_dt_blocks<Q, 512><<<grid, nt, smem, st>>>(g, nl, rec, M, D, hist);
    else k_dt_blocks<Q, 256><<<grid, nt, smem, st>>>(g, nl, rec, M, D, hist);
    CK(cudaGetLastError());
    return 0;
}

// the transform kernels of every q, for a runtime q
template <template <int> class F, class... A>
int dt_for_q(int q, A... a)
{
    switch (q) {
    case 2: return F<2>::run(a...);   case 3: return F<3>::run(a...);   case 4: return F<4>::run(a...);
    case 5: return F<5>::run(a...);   case 6: return F<6>::run(a...);   case 7: return F<7>::run(a...);
    case 8: return F<8>::run(a...);   case 9: return F<9>::run(a...);   case 10: return F<10>::run(a...);
    case 11: return F<11>::run(a...); case 12: return F<12>::run(a...); case 13: return F<13>::run(a...);
    case 14: return F<14>::run(a...); case 15: return F<15>::run(a...); case 16: return F<16>::run(a...);
    default: return COV_EINVAL;
    }
}

template <int Q> struct DtAttrs {
    static int run()
    {
        if (cudaFuncSetAttribute(k_dt_low<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_TILE_BIG) != cudaSuccess ||
            cudaFuncSetAttribute(k_dt_high<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_STRIP_MAX) != cudaSuccess ||
            cudaFuncSetAttribute(k_dt_tiles<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_TILES_SMEM) != cudaSuccess)
            return -(100 + (int)cudaGetLastError());
        return 0;
    }
};
template <int Q> struct DtTiles {
    static int run(int grid, int nt, size_t smem, cudaStream_t st, const uint8_t *code, int M, DtGeom g, int nl,
                   uint2 *rec, uint8_t *D, unsigned long long *hist)
    {
        if (M > 0) {
            k_dt_records<Q><<<std::min(1024, (M + 255) / 256), 256, 0, st>>>(code, M, g, nl, rec);
            CK(cudaGetLastError());
        }
        k_dt_tiles<Q><<<grid, nt, smem, st>>>(g, nl, rec, M, D, hist);
        CK(cudaGetLastError());
        return 0;
    }
};
template <int Q> struct DtLow {
    static int run(int grid, int nt, size_t smem, cudaStream_t st, DtGeom g, int k, const uint32_t *bm,
                   uint8_t *D, unsigned long long *hist)
    {
        k_dt_low<Q><<<grid, nt, smem, st>>>(g, k, bm, D, hist);
        return 0;
    }
};
template <int Q> struct DtHigh {
    static int run(int grid, size_t smem, cudaStream_t st, DtGeom g, int j0, int gsz, int lw, int last,
                   uint8_t *D, unsigned long long *hist)
    {
        k_dt_high<Q><<<grid, DT_NT, smem, st>>>(g, j0, gsz, lw, last, D, hist);
        return 0;
    }
};

__global__ void k_count_above(const uint8_t *__restrict__ D, uint32_t N, int R, unsigned long long *out)
{
    unsigned long long c = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x)
        c += D[x] > R;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ------------------------------------------------ coverage multiplicity ----
// the tiles' records of a code given as digits (one outside the alphabet is
// taken as the largest digit, so that every mark stays within its tile)
__global__ void k_count_records(const uint8_t *__restrict__ code, int M, int q, int n, int nh, int nl, uint2 *mid,
                                uint32_t *hi)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const uint8_t *c = code + (size_t)i * n;
        bt_record(i, q, n, nh, nl, mid, hi, [&](int j) { return (uint32_t)min((int)c[j], q - 1); });
    }
}

// the same of word indices
__global__ void k_count_records_idx(const uint32_t *__restrict__ idx, int M, int q, int n, int nh, int nl, uint2 *mid,
                                    uint32_t *hi)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        uint64_t pk = 0;
        uint32_t x = idx[i];
        for (int j = n - 1; j >= 0; j--) { pk |= (uint64_t)(x % (uint32_t)q) << (4 * j); x /= (uint32_t)q; }
        bt_record(i, q, n, nh, nl, mid, hi, [&](int j) { return (uint32_t)cov_nib(pk, j); });
    }
}

struct CountGeom {
    int q, n, R, M, nh, nl;
    uint32_t tw;                       // q^nl words per tile
    uint32_t vcum[COV_MAXN + 2];
};

// cnt[x] = #{i : d(x, c_i) <= R} saturated at 65535 (the cnt[] of
// covsearch2e.c:958-967, the OUT=2 map of cov/gemm2/dct.cu:360-411), one CTA
// per tile (cov_tiles.cuh).
template <int Q>
__global__ void __launch_bounds__(BT_NT) k_count_tiles(CountGeom g, BtCode code, uint16_t *cnt)
{
    extern __shared__ __align__(16) uint32_t ct_sm[];
    const BtTile tl = bt_layout(g.q, g.n, g.tw);
    bt_mark_tile<Q>(ct_sm, tl, blockIdx.x, g.q, g.n, g.R, g.M, code, g.nh, g.nl, g.vcum,
                    [](uint32_t) { return 1u; });
    uint16_t *out = cnt + (size_t)blockIdx.x * g.tw;
    const uint32_t *tile = ct_sm + tl.a0;
    // whole 32-bit words between the first and the last 4-byte boundary
    const uint32_t head = (uint32_t)(reinterpret_cast<uintptr_t>(out) >> 1) & 1u;
    const uint32_t np = (g.tw - head) >> 1;
    for (uint32_t k = threadIdx.x; k < np; k += BT_NT)
        *reinterpret_cast<uint32_t *>(out + head + 2 * k) =
            min(tile[head + 2 * k], 65535u) | (min(tile[head + 2 * k + 1], 65535u) << 16);
    if (threadIdx.x == 0 && head) out[0] = (uint16_t)min(tile[0], 65535u);
    if (threadIdx.x == 1 && ((g.tw - head) & 1u)) out[g.tw - 1] = (uint16_t)min(tile[g.tw - 1], 65535u);
}

// The same sums as whole 32-bit words: map[x] = #{i : d(x, c_i) <= R}, or
// that many less than before.
template <int Q>
__global__ void __launch_bounds__(BT_NT) k_count_tiles_map(CountGeom g, BtCode code, int32_t *map, int subtract)
{
    extern __shared__ __align__(16) uint32_t ct_sm[];
    const BtTile tl = bt_layout(g.q, g.n, g.tw);
    bt_mark_tile<Q>(ct_sm, tl, blockIdx.x, g.q, g.n, g.R, g.M, code, g.nh, g.nl, g.vcum,
                    [](uint32_t) { return 1u; });
    int32_t *out = map + (size_t)blockIdx.x * g.tw;
    const uint32_t *tile = ct_sm + tl.a0;
    if (subtract) {
#pragma unroll 4
        for (uint32_t k = threadIdx.x; k < g.tw; k += BT_NT) out[k] -= (int32_t)tile[k];
    } else {
        for (uint32_t k = threadIdx.x; k < g.tw; k += BT_NT) out[k] = (int32_t)tile[k];
    }
}

// ------------------------------------------------------------ finisher ----
struct FinishGeom {
    int q, n, R, M;
    uint32_t N;
    uint32_t pw[COV_MAXN];             // q^(n-1-j)
    uint32_t ngroups;                  // ball groups of radius <= R (cov_tiles.cuh, nh = 0)
};

__device__ __forceinline__ uint64_t fin_xorshift(uint64_t r)
{
    r ^= r << 13;
    r ^= r >> 7;
    r ^= r << 17;
    return r;
}

// +1 (saturating) over the ball of the packed word pc into cnt; all threads
__device__ void fin_mark(const FinishGeom &g, uint16_t *cnt, uint64_t pc, const uint64_t *items,
                         const uint8_t *last)
{
    uint32_t base = 0;
    for (int j = 0; j < g.n; j++) base += (uint32_t)cov_nib(pc, j) * g.pw[j];
    for (uint32_t it = threadIdx.x; it < g.ngroups; it += blockDim.x) {
        uint64_t sp = items[it];
        int off = (int)base;
        while (sp) {
            const int j = (__ffsll((long long)sp) - 1) >> 2;
            const int dig = (int)((sp >> (4 * j)) & 15u) - 1;
            sp &= ~(15ull << (4 * j));
            const int cj = cov_nib(pc, j);
            off += (dig + (dig >= cj) - cj) * (int)g.pw[j];
        }
        const int lj = last[it];
        if (lj == 0xff) {
            if (cnt[off] != 0xffffu) cnt[off]++;
        } else {
            const int step = (int)g.pw[lj], cj = cov_nib(pc, lj);
            int o2 = off - cj * step;
            for (int v = 0; v < g.q; v++, o2 += step)
                if (v != cj && cnt[o2] != 0xffffu) cnt[o2]++;
        }
    }
}

// Top-up of covcount (cov/engine/covcount.c:163-195), one CTA: words m0..M-1
// of code[] (packed) are chosen in order -- the first of 64 xorshift64
// draws (seeded 88172645463325252 ^ m0) that is still uncovered, else the
// first uncovered word from the scan position on, else any draw not yet in
// the code -- and each one's ball is marked before the next is chosen.
// Words of one ball are distinct, so the marking needs no atomics.
__global__ void __launch_bounds__(512) k_topup(FinishGeom g, uint16_t *cnt, uint64_t *code, int m0,
                                               const uint64_t *__restrict__ items,
                                               const uint8_t *__restrict__ last)
{
    __shared__ uint64_t draw_st[64];
    __shared__ uint32_t draw_x[64];
    __shared__ unsigned hit[2];
    __shared__ uint64_t s_rs;
    __shared__ long long s_w, s_scan;
    __shared__ int s_dup;
    __shared__ uint64_t s_new;
    if (threadIdx.x == 0) { s_rs = 88172645463325252ull ^ (uint64_t)m0; s_scan = 0; }
    __syncthreads();
    for (int m = m0; m < g.M; m++) {
        if (threadIdx.x == 0) {
            uint64_t r = s_rs;
            for (int t = 0; t < 64; t++) { r = fin_xorshift(r); draw_st[t] = r; draw_x[t] = (uint32_t)(r % g.N); }
        }
        __syncthreads();
        if (threadIdx.x < 64) {
            const unsigned b = __ballot_sync(0xffffffffu, cnt[draw_x[threadIdx.x]] == 0);
            if ((threadIdx.x & 31) == 0) hit[threadIdx.x >> 5] = b;
        }
        __syncthreads();
        int f = -1;
        if (hit[0]) f = __ffs(hit[0]) - 1;
        else if (hit[1]) f = 32 + __ffs(hit[1]) - 1;
        long long w = -1;
        if (f >= 0) {
            w = draw_x[f];
        } else {
            // first zero at or after the scan position, in chunks of the block
            for (long long x0 = s_scan; x0 < (long long)g.N && w < 0; x0 += blockDim.x) {
                const long long x = x0 + threadIdx.x;
                const int z = x < (long long)g.N && cnt[x] == 0;
                const int any = __syncthreads_or(z);
                if (any) {
                    if (threadIdx.x == 0) s_w = 0x7fffffffffffffffll;
                    __syncthreads();
                    if (z) atomicMin((unsigned long long *)&s_w, (unsigned long long)x);
                    __syncthreads();
                    w = s_w;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_rs = f >= 0 ? draw_st[f] : draw_st[63];
            s_scan = f >= 0 ? s_scan : (w >= 0 ? w : (long long)g.N);
        }
        __syncthreads();
        if (w >= 0) {
            if (threadIdx.x == 0) {
                uint64_t pk = 0;
                uint32_t y = (uint32_t)w;
                for (int j = g.n - 1; j >= 0; j--) { pk |= (uint64_t)(y % (uint32_t)g.q) << (4 * j); y /= (uint32_t)g.q; }
                s_new = pk;
            }
        } else {
            // everything covered: any draw that is not yet a codeword
            for (;;) {
                if (threadIdx.x == 0) {
                    s_rs = fin_xorshift(s_rs);
                    uint32_t y = (uint32_t)(s_rs % g.N);
                    uint64_t pk = 0;
                    for (int j = g.n - 1; j >= 0; j--) { pk |= (uint64_t)(y % (uint32_t)g.q) << (4 * j); y /= (uint32_t)g.q; }
                    s_new = pk;
                    s_dup = 0;
                }
                __syncthreads();
                for (int i = threadIdx.x; i < m; i += blockDim.x)
                    if (code[i] == s_new) s_dup = 1;
                __syncthreads();
                if (!s_dup) break;
                __syncthreads();
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) code[m] = s_new;
        fin_mark(g, cnt, s_new, items, last);
        __syncthreads();
    }
}

__global__ void k_count_zero16(const uint16_t *cnt, uint32_t N, unsigned long long *out)
{
    unsigned long long c = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x)
        c += cnt[x] == 0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ============================================================ host ========
namespace {

long long ipw(long long b, int e) { long long r = 1; while (e-- > 0) r *= b; return r; }

int geom(int q, int n, DtGeom &g)
{
    if (q < 2 || q > 16 || n < 1 || n > 16) return COV_EINVAL;
    long long N = ipw(q, n);
    if (N >= (1LL << 32) - 1) return COV_EINVAL;
    g.q = q; g.n = n; g.N = (uint32_t)N; g.inf = n + 1;
    for (int k = 0; k <= COV_MAXN; k++) g.pw[k] = (uint32_t)std::min<long long>(ipw(q, k), 0xffffffffLL);
    return 0;
}

// Scratch of the verification calls: stream-ordered allocations from a memory
// pool of the library's own, per device, that keeps at most SCRATCH_KEEP bytes
// between calls (more goes back at the next synchronisation).  The default
// pool gives everything back at each, and a call that maps memory anew takes
// 100 to 200 us longer; so did a cudaMalloc and cudaFree for each buffer
// (6^6: 213 us for a transform of 11).  A pool reserves 32 MB at a time and
// goes by what it has reserved, so that a limit of 16 MB kept nothing over a
// device synchronisation: a lone call took 264 us, and takes 62 with two such
// pieces kept.
#define SCRATCH_KEEP (64ull << 20)

int scratch_alloc(void **p, size_t bytes, cudaStream_t st)
{
    static cudaMemPool_t pools[COV_MAX_DEVICES];
    static std::mutex m;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= COV_MAX_DEVICES) return COV_ENODEV;
    {
        std::lock_guard<std::mutex> hold(m);
        if (!pools[dev]) {
            cudaMemPoolProps props;
            memset(&props, 0, sizeof props);
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaMemPool_t pool = nullptr;
            // the call may be one that a stream captures: making a pool is no
            // work of the stream, but is refused unless the thread's mode is
            // relaxed, and the capture is lost
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            CK(cudaThreadExchangeStreamCaptureMode(&mode));
            cudaError_t e = cudaMemPoolCreate(&pool, &props);
            unsigned long long keep = SCRATCH_KEEP;
            if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            CK(cudaThreadExchangeStreamCaptureMode(&mode));
            CK(e);
            pools[dev] = pool;
        }
    }
    if (cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), pools[dev], st) != cudaSuccess) {
        cudaGetLastError();
        return COV_ENOMEM;
    }
    return 0;
}

CovDeviceFlags g_dt_attr;   // shared-memory opt-in of the transform kernels, per device
CovDeviceFlags g_ct_attr;   // the same for the tile count

// the tile count of the alphabet size q (BT_Q_LIST: a kernel of its own)
void ct_launch(const CountGeom &g, BtCode code, uint16_t *cnt, cudaStream_t st)
{
    const unsigned grid = (unsigned)ipw(g.q, g.nh);
    const size_t smem = bt_smem_bytes(g.q, g.n, g.tw);
    switch (g.n < 2 ? 0 : g.q) {
#define CT_LAUNCH_Q(QQ) case QQ: k_count_tiles<QQ><<<grid, BT_NT, smem, st>>>(g, code, cnt); break;
    BT_Q_LIST(CT_LAUNCH_Q)
#undef CT_LAUNCH_Q
    default: k_count_tiles<0><<<grid, BT_NT, smem, st>>>(g, code, cnt); break;
    }
}

// the same into a map
void ct_launch_map(const CountGeom &g, BtCode code, int32_t *map, int subtract, cudaStream_t st)
{
    const unsigned grid = (unsigned)ipw(g.q, g.nh);
    const size_t smem = bt_smem_bytes(g.q, g.n, g.tw);
    switch (g.n < 2 ? 0 : g.q) {
#define CT_LAUNCH_Q(QQ) case QQ: k_count_tiles_map<QQ><<<grid, BT_NT, smem, st>>>(g, code, map, subtract); break;
    BT_Q_LIST(CT_LAUNCH_Q)
#undef CT_LAUNCH_Q
    default: k_count_tiles_map<0><<<grid, BT_NT, smem, st>>>(g, code, map, subtract); break;
    }
}

// the tile geometry of a count of M codewords
CountGeom count_geom(int q, int n, int R, int M)
{
    CountGeom g;
    memset(&g, 0, sizeof g);
    g.q = q; g.n = n; g.R = R; g.M = M;
    bt_geom(q, n, R, M, std::max(1, cov_sm_count()), &g.nh, &g.nl);
    g.tw = (uint32_t)ipw(q, g.nl);
    bt_vcum_h(q, n, R, g.nl, g.vcum);
    return g;
}

int ct_attrs()
{
    int dev = 0;
    if (g_ct_attr.done(dev)) return 0;
    CK(cudaFuncSetAttribute(k_count_tiles<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            BT_SMEM_MAX));
    CK(cudaFuncSetAttribute(k_count_tiles_map<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, BT_SMEM_MAX));
#define CT_ATTR_Q(QQ) \
    CK(cudaFuncSetAttribute(k_count_tiles<QQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, BT_SMEM_MAX)); \
    CK(cudaFuncSetAttribute(k_count_tiles_map<QQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, BT_SMEM_MAX));
    BT_Q_LIST(CT_ATTR_Q)
#undef CT_ATTR_Q
    g_ct_attr.set(dev);
    return 0;
}

// How a transform runs: by tiles from the code alone (k_dt_tiles) or by the
// bitmap and sweeps of the word array (k_dt_low, k_dt_high).
struct DtPlan {
    bool tiles, blocks;          // blocks: tiles by k_dt_blocks
    int nl, nt, grid;
    size_t smem;
    size_t scratch;              // bytes of device scratch: the code's records, or its bitmap
};

// The tile form costs M code marks a tile, so the rule compares estimates in
// SM cycles.  A tile takes about 25 lane-instructions a codeword (12 more
// where the threads cannot keep them), 11 a line and pass, 4 a word of
// output, at 64 lanes a cycle, and a latency chain of some 500 cycles a
// barrier; the number of low digits with the least estimate is taken (of the
// seven cells timed at every number it is the best or within 6 % of it).  The
// sweep form's side is measured: 4.2 ps a word (8^10: 4.5 ms) after three
// launches.  Measured, sweeps against lines against blocks (q = 5..8: 30
// lane-instructions a codeword and a block's pass, 2.5 to 5 a word of output):
// 8^10 M 2549 4505, 686, 367 us; 7^10 M 163 1076, 267, 139; 7^9 M 1500 179,
// 57, 40; 7^9 M 30000 179, 85; 6^6 M 41 24.8, 10.6; near the line, 8^7 M
// 30000: sweeps 41.1, lines 41.7.
#define DT_SWEEP_CYCLES_WORD 0.0087
#define DT_SWEEP_CYCLES_MIN 16000.0
DtPlan dt_plan(const DtGeom &g, int M, const uint8_t *D)
{
    DtPlan best{};
    best.scratch = (size_t)((g.N + 31) / 32) * 4;
    double least = DT_SWEEP_CYCLES_MIN + DT_SWEEP_CYCLES_WORD * g.N;
    const double sms = std::max(1, cov_sm_count());
    for (int nl = std::max(1, g.n - 8); nl <= g.n; nl++) {
        const uint32_t T = g.pw[nl], lines = g.pw[nl - 1];
        if ((size_t)lines * 4 > DT_TILES_SMEM) break;
        const int nt = lines > 8192 ? 512 : lines > 256 ? 256 : 128;
        const double tiles = g.N / T;
        const double per_sm = std::min(std::min(1536.0 / nt, 220.0 * 1024 / (lines * 4.0 + 1200)), 32.0);
        const double work = M * (M <= nt * DT_TILES_KEEP ? 25.0 : 37.0) + lines * 11.0 * (nl - 1) + T * 4.0;
        const double waves = std::ceil(tiles / (sms * std::floor(per_sm)));
        const double cyc = tiles * work / (64.0 * sms) + waves * (1500.0 + 500.0 * nl + work / (nt / 4.0));
        if (cyc < least) {
            least = cyc;
            best.tiles = true;
            best.nl = nl;
            best.nt = nt;
            best.smem = (size_t)lines * 4;
            best.grid = (int)std::min(tiles, sms * std::floor(per_sm));
            best.scratch = (size_t)std::max(M, 1) * 8;
        }
    }
    // blocks of two digits (q = 8 stores 16 bytes at a time)
    if (g.q < 5 || g.q > 8 || (g.q == 8 && (reinterpret_cast<uintptr_t>(D) & 15u))) return best;
    for (int nl = std::max(2, g.n - 8); nl <= g.n; nl++) {
        const uint32_t T = g.pw[nl], nblk = T / (uint32_t)(g.q * g.q);
        const size_t smem = (size_t)nblk * (g.q == 5 ? 12 : 20);
        if (smem > DT_BLOCKS_SMEM) break;
        const int nt = nblk <= 64 ? 128 : nblk > 1024 && (g.q == 5 || M > 4096) ? 512 : 256;
        const double tiles = g.N / T;
        const double per_sm = std::min(std::min((nt > 256 ? 1024.0 : 768.0) / nt, 220.0 * 1024 / (smem + 2048.0)), 32.0);
        const double work = M * (M <= nt * DT_TILES_KEEP ? 30.0 : 45.0) + nblk * (30.0 * (nl - 2) + 15.0) +
                            T * (g.q == 8 ? 2.5 : 5.0);
        const double waves = std::ceil(tiles / (sms * std::floor(per_sm)));
        const double cyc = tiles * work / (64.0 * sms) + waves * (2000.0 + 500.0 * (nl - 2) + work / (nt / 4.0));
        if (cyc < least) {
            least = cyc;
            best.tiles = best.blocks = true;
            best.nl = nl;
            best.nt = nt;
            best.smem = smem;
            best.grid = (int)std::min(tiles, sms * std::floor(per_sm));
            best.scratch = (size_t)std::max(M, 1) * 8;
        }
    }
    return best;
}

// the transform on device buffers; hist (device, n+2 entries) may be null,
// and d_D too when the plan is by tiles; scratch: plan.scratch bytes
int dt_run(const DtGeom &g, const DtPlan &plan, const uint8_t *d_code, int M, uint8_t *d_D,
           unsigned long long *d_hist, void *scratch, cudaStream_t st)
{
    int dev = 0;
    if (!g_dt_attr.done(dev)) {
        for (int q = 2; q <= COV_MAXQ; q++) {
            const int rc = dt_for_q<DtAttrs>(q);
            if (rc) return rc;
        }
        for (const void *k : {(const void *)k_dt_blocks<5, 256>, (const void *)k_dt_blocks<6, 256>,
                              (const void *)k_dt_blocks<7, 256>, (const void *)k_dt_blocks<8, 256>,
                              (const void *)k_dt_blocks<5, 512>, (const void *)k_dt_blocks<6, 512>,
                              (const void *)k_dt_blocks<7, 512>, (const void *)k_dt_blocks<8, 512>})
            CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_BLOCKS_SMEM));
        g_dt_attr.set(dev);
    }
    if (plan.blocks) {
        switch (g.q) {
#define DT_BLOCKS_Q(QQ) case QQ: return dt_blocks_launch<QQ>(plan.grid, plan.nt, plan.smem, st, d_code, M, g, plan.nl, \
                                                             (uint2 *)scratch, d_D, d_hist);
        DT_BLOCKS_Q(5) DT_BLOCKS_Q(6) DT_BLOCKS_Q(7) DT_BLOCKS_Q(8)
#undef DT_BLOCKS_Q
        }
    }
    if (plan.tiles)
        return dt_for_q<DtTiles>(g.q, plan.grid, plan.nt, plan.smem, st, d_code, M, g, plan.nl, (uint2 *)scratch,
                                 d_D, d_hist);
    uint32_t *d_bm = (uint32_t *)scratch;
    CK(cudaMemsetAsync(d_bm, 0, (size_t)((g.N + 31) / 32) * 4, st));
    if (M > 0) {
        k_dt_bitmap<<<std::min(1024, (M + 255) / 256), 256, 0, st>>>(d_code, M, g, d_bm);
        CK(cudaGetLastError());
    }
    // low group: as many axes as fit a tile
    const long long q4 = (g.q + 3) / 4 * 4;      // padded bytes of one lowest-axis line
    auto low_bytes = [&](int kk) { return (long long)g.pw[kk] / g.q * q4; };
    // HBM sweeps of the strip passes after a low tile of kk axes
    auto strip_sweeps = [&](int kk) {
        int sw = 0, j = kk;
        while (j < g.n) {
            int gz = 0;
            while (j + gz < g.n && (long long)g.pw[gz + 1] * DT_STRIP_W <= DT_STRIP_MAX) gz++;
            j += std::max(gz, 1);
            sw++;
        }
        return sw;
    };
    int k = 1;
    while (k < g.n && low_bytes(k + 1) <= DT_TILE_MAX) k++;
    // a bigger tile (one CTA per SM, twice the threads) only where it saves a sweep
    int kb = k;
    while (kb < g.n && low_bytes(kb + 1) <= DT_TILE_BIG) kb++;
    const bool big = strip_sweeps(kb) < strip_sweeps(k);
    if (big) k = kb;
    const int sms = std::max(1, cov_sm_count());
    const uint32_t ntile = g.N / g.pw[k];
    {
        int grid = (int)std::min<uint32_t>(ntile, (uint32_t)sms * (big ? 1 : 4));
        dt_for_q<DtLow>(g.q, grid, big ? DT_NT_BIG : DT_NT, (size_t)low_bytes(k), st, g, k,
                        (const uint32_t *)d_bm, d_D, d_hist);
        CK(cudaGetLastError());
    }
    // high groups
    int j0 = k;
    while (j0 < g.n) {
        int gsz = 0;
        while (j0 + gsz < g.n && (long long)g.pw[gsz + 1] * DT_STRIP_W <= DT_STRIP_MAX) gsz++;
        if (gsz == 0) return COV_EINVAL;
        int last = (j0 + gsz == g.n);
        const uint32_t s = g.pw[j0];
        // widest power-of-two strip (>= DT_STRIP_W bytes) the shared memory
        // holds for these rows, but no wider than the group's stride needs
        int lw = 0;
        while ((long long)g.pw[gsz] * (DT_STRIP_W << (lw + 1)) <= DT_STRIP_MAX &&
               (uint32_t)(DT_STRIP_W << lw) < s)
            lw++;
        const uint32_t W = (uint32_t)DT_STRIP_W << lw;
        const unsigned long long tiles = (unsigned long long)(g.N / (g.pw[gsz] * s)) * ((s + W - 1) / W);
        int grid = (int)std::min<unsigned long long>(tiles, (unsigned long long)sms * 4);
        dt_for_q<DtHigh>(g.q, grid, (size_t)g.pw[gsz] * W, st, g, j0, gsz, lw, last, d_D, d_hist);
        CK(cudaGetLastError());
        j0 += gsz;
    }
    return 0;
}

}  // namespace

// the records of the m listed words and the geometry of their count
static int words_records(int q, int n, int R, const uint32_t *d_idx, int m, uint2 *rec, cudaStream_t st, CountGeom &g,
                         BtCode &code)
{
    int rc = ct_attrs();
    if (rc) return rc;
    g = count_geom(q, n, std::min(R, n), m);
    uint32_t *hi = (uint32_t *)(rec + m);
    code = BtCode{hi, rec};
    if (m > 0) {
        k_count_records_idx<<<std::min(1024, (m + 127) / 128), 128, 0, st>>>(d_idx, m, q, n, g.nh, g.nl, rec, hi);
        CK(cudaGetLastError());
    }
    return COV_OK;
}

int cov_count_words(int q, int n, int R, const uint32_t *d_idx, int m, uint16_t *cnt, uint2 *rec, cudaStream_t st)
{
    CountGeom g;
    BtCode code;
    int rc = words_records(q, n, R, d_idx, m, rec, st, g, code);
    if (rc) return rc;
    ct_launch(g, code, cnt, st);
    CK(cudaGetLastError());
    return COV_OK;
}

int cov_count_words_map(int q, int n, int R, const uint32_t *d_idx, int m, int32_t *map, int subtract, uint2 *rec,
                        cudaStream_t st)
{
    CountGeom g;
    BtCode code;
    int rc = words_records(q, n, R, d_idx, m, rec, st, g, code);
    if (rc) return rc;
    ct_launch_map(g, code, map, subtract, st);
    CK(cudaGetLastError());
    return COV_OK;
}

extern "C" {

int cov_mindist_dev(int32_t q, int32_t n, const uint8_t *d_code, int32_t M, uint8_t *d_dist, void *stream)
{
    DtGeom g;
    int rc = geom(q, n, g);
    if (rc) return rc;
    if (M < 0 || (M > 0 && !d_code) || !d_dist) return COV_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    const DtPlan plan = dt_plan(g, M, d_dist);
    void *scratch = nullptr;
    rc = scratch_alloc(&scratch, plan.scratch, st);
    if (rc) return rc;
    rc = dt_run(g, plan, d_code, M, d_dist, nullptr, scratch, st);
    cudaFreeAsync(scratch, st);
    return rc;
}

// ---------------------------------------------------------------------------
// Allocation-free distance transform.
//
// For callers that must not allocate device memory themselves: a host runtime
// whose device memory is entirely owned by another allocator (for example a
// framework's caching allocator that has reserved the whole GPU), or code
// that runs where an allocation would break the surrounding contract (inside
// an out-of-memory handler).  The one scratch buffer the transform needs --
// the codewords' records of the tile forms, or the bitmap of codeword
// positions of the sweeps -- lives in a file-scope device array instead of
// being allocated per call.
//
//  * Limit: q^n <= COV_DT_STATIC_MAX_WORDS (2^26 words, whose bitmap is the
//    8 MiB of the array, which every GPU that loads the library keeps until
//    the process exits).  A code with more records than the array holds (8
//    bytes each, 2^20 codewords) takes the sweeps.
//  * The first call on a device looks up the array's device address
//    (cudaGetSymbolAddress, with that device current) and caches it.
//  * Every call writes the same array anew before it reads it: two calls
//    whose work overlaps on the GPU (different streams, no ordering) race.
#define COV_DT_STATIC_MAX_WORDS (1u << 26)
#define COV_DT_STATIC_MAX_DEVICES 64

static __device__ __align__(256) uint32_t g_dt_static_bitmap[COV_DT_STATIC_MAX_WORDS / 32];
static uint32_t *g_dt_static_addr[COV_DT_STATIC_MAX_DEVICES];   // per device, host side

int cov_mindist_dev_static(int32_t q, int32_t n, const uint8_t *d_code, int32_t M, uint8_t *d_dist, void *stream)
{
    DtGeom g;
    int rc = geom(q, n, g);
    if (rc) return rc;
    if (g.N > COV_DT_STATIC_MAX_WORDS) {
        fprintf(stderr, "cov_mindist_dev_static: q^n = %u words exceeds the %u-word limit of the static scratch\n",
                g.N, COV_DT_STATIC_MAX_WORDS);
        return COV_ERANGE;
    }
    if (M < 0 || (M > 0 && !d_code) || !d_dist) return COV_EINVAL;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= COV_DT_STATIC_MAX_DEVICES) return COV_ENODEV;
    if (!g_dt_static_addr[dev]) {
        // the array's name is only a host-side stand-in: ask the runtime for
        // its address on the current device
        void *ptr = nullptr;
        CK(cudaGetSymbolAddress(&ptr, g_dt_static_bitmap));
        g_dt_static_addr[dev] = (uint32_t *)ptr;
    }
    DtPlan plan = dt_plan(g, M, d_dist);
    if (plan.scratch > sizeof g_dt_static_bitmap) plan = DtPlan{};       // more codewords than the array has records
    return dt_run(g, plan, d_code, M, d_dist, nullptr, g_dt_static_addr[dev], (cudaStream_t)stream);
}

int64_t cov_count_above_dev(int32_t q, int32_t n, const uint8_t *d_dist, int32_t R, void *stream)
{
    DtGeom g;
    int rc = geom(q, n, g);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long *d_c = nullptr, h = 0;
    rc = scratch_alloc((void **)&d_c, 8, st);
    if (rc) return rc;
    cudaError_t e = cudaMemsetAsync(d_c, 0, 8, st);
    k_count_above<<<std::max(1, cov_sm_count()) * 8, 256, 0, st>>>(d_dist, g.N, R, d_c);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d_c, 8, cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d_c, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    CK(e);
    return (int64_t)h;
}

int cov_mindist(int32_t q, int32_t n, const uint8_t *code, int32_t M, uint8_t *dist, int64_t *hist,
                int32_t *radius)
{
    DtGeom g;
    int rc = geom(q, n, g);
    if (rc) return rc;
    if (M < 0 || (M > 0 && !code)) return COV_EINVAL;
    for (long long i = 0; i < (long long)M * n; i++) if (code[i] >= q) return COV_EINVAL;
    cudaStream_t st = nullptr;
    const DtPlan plan = dt_plan(g, M, nullptr);   // D will be 256-byte aligned
    const bool want_D = dist || !plan.tiles;      // the sweeps work in D; the tiles need none for the histogram
    // one allocation: the histogram, the transform's scratch, the code, D
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t hb = up(8 * (COV_MAXN + 2)), sb = up(plan.scratch), cb = up((size_t)std::max(M, 1) * n);
    uint8_t *buf = nullptr;
    rc = scratch_alloc((void **)&buf, hb + sb + cb + (want_D ? (size_t)g.N : 0), st);
    if (rc) return rc;
    unsigned long long *d_h = (unsigned long long *)buf;
    uint8_t *d_code = buf + hb + sb, *d_D = want_D ? d_code + cb : nullptr;
    auto done = [&](int r) { cudaFreeAsync(buf, st); return r; };
    if (M > 0 && cudaMemcpyAsync(d_code, code, (size_t)M * n, cudaMemcpyHostToDevice, st) != cudaSuccess) return done(-100);
    if (cudaMemsetAsync(d_h, 0, 8 * (COV_MAXN + 2), st) != cudaSuccess) return done(-100);
    rc = dt_run(g, plan, d_code, M, d_D, d_h, buf + hb, st);
    if (rc) return done(rc);
    unsigned long long hh[COV_MAXN + 2];
    cudaError_t e = cudaMemcpyAsync(hh, d_h, 8 * (COV_MAXN + 2), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && dist) e = cudaMemcpyAsync(dist, d_D, g.N, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return done(-(100 + (int)e));
    int rad = 0;
    for (int v = 0; v <= n + 1; v++) {
        if (hist) hist[v] = (int64_t)hh[v];
        if (hh[v]) rad = v;
    }
    if (radius) *radius = rad;
    return done(COV_OK);
}

int cov_verify(int32_t q, int32_t n, int32_t R, const uint8_t *code, int32_t M, int64_t *uncovered)
{
    if (R < 0) return COV_EINVAL;
    int64_t hist[COV_MAXN + 2];
    int rc = cov_mindist(q, n, code, M, nullptr, hist, nullptr);
    if (rc) return rc;
    int64_t u = 0;
    for (int v = R + 1; v <= n + 1; v++) u += hist[v];
    if (uncovered) *uncovered = u;
    return COV_OK;
}

int cov_count_dev(int32_t q, int32_t n, int32_t R, const uint8_t *d_code, int32_t M, uint16_t *d_cnt,
                  void *stream)
{
    DtGeom dg;
    int rc = geom(q, n, dg);
    if (rc) return rc;
    if (R < 0 || M < 0 || M > 65535 || (M > 0 && !d_code) || !d_cnt) return COV_EINVAL;
    if (R > n) R = n;
    cudaStream_t st = (cudaStream_t)stream;
    rc = ct_attrs();
    if (rc) return rc;
    const CountGeom g = count_geom(q, n, R, M);
    void *tmp = nullptr;
    rc = scratch_alloc(&tmp, (size_t)std::max(M, 1) * BT_REC_BYTES, st);
    if (rc) return rc;
    uint2 *mid = (uint2 *)tmp;
    uint32_t *hi = (uint32_t *)(mid + M);
    if (M > 0) {
        k_count_records<<<std::min(1024, (M + 127) / 128), 128, 0, st>>>(d_code, M, q, n, g.nh, g.nl, mid, hi);
    }
    ct_launch(g, BtCode{hi, mid}, d_cnt, st);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(tmp, st);
    CK(e);
    return COV_OK;
}

// The finisher of cov/engine/covcount.c: de-duplicate the m words (first
// occurrences kept), top them up to M distinct words and count the
// uncovered words of the result.  fast: top-up in base-q counting order, no
// coverage (uncovered = -1).
int cov_finish(int32_t q, int32_t n, int32_t R, int32_t M, const uint8_t *code, int32_t m, int32_t fast,
               uint8_t *out, int32_t *words, int64_t *uncovered)
{
    DtGeom dg;
    int rc = geom(q, n, dg);
    if (rc) return rc;
    if (R < 0 || M < 1 || m < 0 || (m > 0 && !code) || !out) return COV_EINVAL;
    if ((long long)M > (long long)dg.N) return COV_EINVAL;           // no M distinct words exist
    if (R > n) R = n;
    for (long long i = 0; i < (long long)m * n; i++) if (code[i] >= q) return COV_EINVAL;
    std::vector<uint64_t> pk;
    {
        pk.reserve((size_t)std::min(m, M));
        // covcount reads at most M words, then drops the repeats among them
        for (int i = 0; i < std::min(m, M); i++) {
            uint64_t v = 0;
            for (int j = 0; j < n; j++) v |= (uint64_t)code[(size_t)i * n + j] << (4 * j);
            if (std::find(pk.begin(), pk.end(), v) == pk.end()) pk.push_back(v);
        }
    }
    const int m0 = (int)pk.size();
    auto unpack = [&](const std::vector<uint64_t> &v) {
        for (int i = 0; i < M; i++)
            for (int j = 0; j < n; j++) out[(size_t)i * n + j] = (uint8_t)((v[i] >> (4 * j)) & 15u);
    };
    if (fast) {
        // base-q counting order, skipping words already present
        std::vector<uint64_t> v = pk;
        for (uint32_t x = 0; (int)v.size() < M; x++) {
            uint64_t w = 0;
            uint32_t y = x;
            for (int j = n - 1; j >= 0; j--) { w |= (uint64_t)(y % (uint32_t)q) << (4 * j); y /= (uint32_t)q; }
            if (std::find(v.begin(), v.end(), w) == v.end()) v.push_back(w);
        }
        unpack(v);
        if (words) *words = M;
        if (uncovered) *uncovered = -1;
        return COV_OK;
    }
    if (dg.N > 1200000000u) return COV_ERANGE;                        // covcount's limit without --fast
    rc = ct_attrs();
    if (rc) return rc;
    // tile count of the deduplicated words
    const CountGeom g = count_geom(q, n, R, m0);
    std::vector<uint8_t> blast;
    // whole-ball groups for the top-up (no high digits)
    uint32_t bcum[COV_MAXN + 2];
    std::vector<uint64_t> bitems = bt_items_h(q, n, R, 0, bcum, blast);
    FinishGeom fg;
    memset(&fg, 0, sizeof fg);
    fg.q = q; fg.n = n; fg.R = R; fg.M = M; fg.N = dg.N;
    for (int j = 0; j < n; j++) fg.pw[j] = dg.pw[n - 1 - j];
    fg.ngroups = bcum[std::min(R, n)];
    const size_t trb = ((size_t)m0 * BT_REC_BYTES + 7) / 8 * 8;
    const size_t bib = bitems.size() * 8, blb = (blast.size() + 7) / 8 * 8;
    const size_t cb = ((size_t)dg.N * 2 + 15) / 16 * 16;
    char *buf = nullptr;
    if (cudaMalloc(&buf, trb + bib + blb + (size_t)M * 8 + cb + 16) != cudaSuccess) {
        cudaGetLastError();
        return COV_ENOMEM;
    }
    uint64_t *d_bi = (uint64_t *)(buf + trb);
    uint8_t *d_bl = (uint8_t *)(buf + trb + bib);
    uint64_t *d_code = (uint64_t *)(buf + trb + bib + blb);
    uint16_t *d_cnt = (uint16_t *)(buf + trb + bib + blb + (size_t)M * 8);
    unsigned long long *d_z = (unsigned long long *)(buf + trb + bib + blb + (size_t)M * 8 + cb);
    auto done = [&](int r) { cudaFree(buf); return r; };
    cudaError_t e = cudaSuccess;
    e = cudaMemcpy(d_bi, bitems.data(), bib, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d_bl, blast.data(), blast.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && m0 > 0) e = cudaMemcpy(d_code, pk.data(), (size_t)m0 * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(d_z, 0, 8);
    if (e != cudaSuccess) return done(-(100 + (int)e));
    const BtCode rec = bt_records(d_code, m0, q, n, g.nh, g.nl, buf, 0);
    ct_launch(g, rec, d_cnt, 0);
    e = cudaGetLastError();
    if (e == cudaSuccess && m0 < M) {
        k_topup<<<1, 512>>>(fg, d_cnt, d_code, m0, d_bi, d_bl);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        k_count_zero16<<<std::max(1, cov_sm_count()) * 4, 256>>>(d_cnt, dg.N, d_z);
        e = cudaGetLastError();
    }
    std::vector<uint64_t> v((size_t)M);
    unsigned long long z = 0;
    if (e == cudaSuccess) e = cudaMemcpy(v.data(), d_code, (size_t)M * 8, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&z, d_z, 8, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return done(-(100 + (int)e));
    unpack(v);
    if (words) *words = M;
    if (uncovered) *uncovered = (int64_t)z;
    return done(COV_OK);
}

int cov_count(int32_t q, int32_t n, int32_t R, const uint8_t *code, int32_t M, uint16_t *cnt,
              int64_t *uncovered)
{
    DtGeom g;
    int rc = geom(q, n, g);
    if (rc) return rc;
    if (R < 0 || M < 0 || M > 65535 || (M > 0 && !code)) return COV_EINVAL;
    for (long long i = 0; i < (long long)M * n; i++) if (code[i] >= q) return COV_EINVAL;
    uint8_t *d_code = nullptr;
    uint16_t *d_cnt = nullptr;
    const size_t nb = ((size_t)g.N + 1) / 2 * 4;     // whole 32-bit pairs
    if (cudaMalloc(&d_code, (size_t)std::max(M, 1) * n) != cudaSuccess ||
        cudaMalloc(&d_cnt, nb) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(d_code); cudaFree(d_cnt);
        return COV_ENOMEM;
    }
    auto done = [&](int r) { cudaFree(d_code); cudaFree(d_cnt); return r; };
    if (M > 0 && cudaMemcpy(d_code, code, (size_t)M * n, cudaMemcpyHostToDevice) != cudaSuccess) return done(-100);
    rc = cov_count_dev(q, n, R, d_code, M, d_cnt, nullptr);
    if (rc) return done(rc);
    std::vector<uint16_t> tmp;
    uint16_t *h = cnt;
    if (!h) { tmp.resize(g.N); h = tmp.data(); }
    cudaError_t e = cudaMemcpy(h, d_cnt, (size_t)g.N * 2, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return done(-(100 + (int)e));
    if (uncovered) {
        int64_t u = 0;
        for (uint32_t x = 0; x < g.N; x++) u += h[x] == 0;
        *uncovered = u;
    }
    return done(COV_OK);
}

}  // extern "C"
