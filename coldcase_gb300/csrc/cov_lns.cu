// cov_lns.cu -- GB300 (sm_103a) transform engine for the ruin-and-recreate
// search over one cell (q, n, R): the capability of cov/gemm2/gpuchain.py
// and its primitives cov/gemm2/dct.cu, built around two device-side pieces.
//
//  * Maps.  gain(x) = #{y : d(x,y) <= R, cnt[y] == 0} (the words a codeword
//    at x would newly cover) and loss(x) = the same with cnt[y] == 1 (the
//    words only a codeword at x covers) are computed for every x at once as
//    layered counts over 64-bit masks of the marked words, one axis at a
//    time.  The axes are not swept one by one through HBM: the low axes are
//    done on contiguous tiles of q^k words in shared memory, the remaining
//    ones on strips of q^g rows x W words, all int32 layers of a tile at once,
//    and all sweeps but the last go part by part through L2.  The counts of a
//    code come from the verifier's tiles.
//  * Sequences.  The lazy greedy placement (bounds from a gain map, the best
//    bounds re-counted exactly until the best is current, then placed) is one
//    cooperative kernel over the whole GPU with no host round trip between
//    its steps; it counts on masks of the uncovered words, a 64-bit word for
//    the q^b words that share their high digits.  The exact peel (codewords
//    removed in a given order while each covers no word alone) is a
//    persistent kernel on one thread-block cluster: every CTA walks a share
//    of each ball, and they meet at hardware cluster barriers and reduce
//    through distributed shared memory.  The +-1 balls of a list of words
//    commute and run at once.
//
// Words are indexed MSB-first (x = sum_j w_j q^(n-1-j)), as everywhere in
// this library.  Extraction returns positions in increasing index order, and
// every tie is broken by the lower position, so every result is
// deterministic.
#include <cstdio>
#include <climits>
#include <cstring>
#include <vector>
#include <algorithm>
#include <cooperative_groups.h>
#include "cov_common.cuh"
#include "cov_tiles.cuh"
#include "cov_map.cuh"
#include "../../include/covgpu.h"

namespace cg = cooperative_groups;

#define LNS_NT 256
#define LNS_HIST_MAX 8192   // bins of cov_lns_map_hist (one shared-memory counter each)
#define SEQ_NT 512
#define SEQ_CL 8                    // CTAs of the sequence cluster
#define CAND_CAP (1 << 17)          // candidate bounds kept on the device per refresh
#define GREEDY_NT 512
#define GREEDY_MAXG 512             // most CTAs of the greedy kernel (one per SM)
#define THR_BINS 1024               // histogram bins behind an extraction threshold
#define MAP_TILES_N 1000000u        // words of the smallest space whose greedy maps may come from tiles
#define MAP_PS_LAUNCH 20e6          // what such a map has to save, ps
#define NOTE_CAP (1 << 16)          // most words whose balls a refresh counts by tiles
#define EXT_CHUNK 8192              // words of one block of an ordered extraction

#define CK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { \
    fprintf(stderr, "covgpu: CUDA error %s at %s:%d\n", cudaGetErrorString(e_), __FILE__, __LINE__); \
    return -(100 + (int)e_); } } while (0)

// state of a sequence launch, read back by the host
struct SeqState {
    long long uncov;             // uncovered words, kept exact through every ball
    long long evals;             // exact ball counts made
    int placed, removed;         // words placed / removed by the launch
    int status;                  // SEQ_*
    int best;                    // greedy: no word's gain is higher at the end of the launch
};

// what a refresh of the greedy's candidates leaves on the device
struct RefreshInfo {
    int top;                     // maximum of the map
    int thr;                     // candidates are the words with map >= thr
    uint32_t found;              // how many there are (saturated)
    uint32_t noted;              // words that k_lns_note wrote
};
enum { SEQ_DONE = 0, SEQ_REFRESH = 1, SEQ_COVERED = 2, SEQ_TARGET = 3, SEQ_GUARD = 5 };

struct cov_lns : MapPlan {
    int q, n, R;
    uint32_t N;
    uint32_t pw[COV_MAXN];          // q^(n-1-j)
    uint16_t *cnt = nullptr;        // coverage multiplicity (saturated)
    int32_t *map_scratch = nullptr;      // the layers between the sweeps of a part (two of them from three groups on)
    int32_t *map_whole = nullptr;        // the layers that reach the last sweep (and word counts: MapPlan)
    int32_t *map = nullptr;         // last map (gain or loss)
    uint64_t *ball = nullptr;       // whole-ball groups (cov_tiles.cuh, no high digits)
    uint8_t *ball_last = nullptr;
    uint32_t ngroups = 0;
    uint32_t *cand = nullptr;       // greedy candidates (positions, increasing)
    int32_t *bound = nullptr;       // their gain bounds
    int nb = 0;                     // digits of a mask block: the most with q^nb <= 64
    uint32_t blk = 1;               // its q^nb words
    uint64_t *um = nullptr;         // uncovered words of every block (built by each greedy call)
    uint64_t *um_map = nullptr;     // the masks of the greedy's last map
    uint32_t *note = nullptr;       // [NOTE_CAP] words, then their tile records
    uint64_t *pball = nullptr;      // ball groups on the n - nb high digits
    uint8_t *pball_last = nullptr;
    uint32_t npgroups = 0;
    uint64_t *lowball = nullptr;    // [blk][nb + 1]: words of a block within 0..nb of each of its words
    unsigned long long *nom = nullptr;   // [2 * GREEDY_MAXG] best keys of the greedy's CTAs
    uint32_t *acc = nullptr;        // [3 * (GREEDY_MAXG + 1)] sums of the greedy's steps, then its barrier
    RefreshInfo *info = nullptr;
    uint32_t *list = nullptr;       // words of a sequence (placed, peeled or applied)
    uint8_t *flag = nullptr;        // per listed word: removed by the peel
    int list_cap = 0;
    SeqState *seq = nullptr;
    void *scratch = nullptr;        // small device buffers of the calls
    size_t scratch_bytes = 0;
    unsigned long long *d_red = nullptr;
};

namespace {

__global__ void k_lns_scatter(int32_t *A0, const uint32_t *idx, int m)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) atomicAdd(&A0[idx[i]], 1);
}

// word counts to saturated counters (the counts at R = 0)
__global__ void k_lns_narrow(const int32_t *A0, uint32_t N, uint16_t *cnt)
{
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x)
        cnt[x] = (uint16_t)min(A0[x], 65535);
}

// the words whose count is target
__global__ void k_lns_indicator(const uint16_t *cnt, int target, uint32_t N, int32_t *out)
{
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x)
        out[x] = (int32_t)(cnt[x] == target);
}

__global__ void k_lns_max(const int32_t *A, uint32_t N, int *out)
{
    int m = INT_MIN;
    const uint32_t step = gridDim.x * blockDim.x;
    unsigned long long x = blockIdx.x * blockDim.x + threadIdx.x;
    for (; x + 7ull * step < N; x += 8ull * step) {
        int v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = __ldcg(&A[x + (unsigned long long)u * step]);
#pragma unroll
        for (int u = 0; u < 8; u++) m = max(m, v[u]);
    }
    for (; x < N; x += step) m = max(m, A[x]);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// histogram of the positive values: value v in bin (min(v,vmax)-1)*nbins/vmax.
// Counted per block in shared memory (the lanes of a warp that share a bin
// add once), then one global add per bin and block: the values of a gain map
// crowd into few bins, where per-element global atomics serialise.  Eight
// loads of a thread are in flight.
__global__ void __launch_bounds__(LNS_NT) k_lns_hist(const int32_t *A, uint32_t N, int nbins, int vmax,
                                                     unsigned long long *hist)
{
    extern __shared__ uint32_t lh[];
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) lh[b] = 0;
    __syncthreads();
    // (v-1)*nbins in 32 bits when it cannot overflow
    const bool narrow = (unsigned long long)vmax * (unsigned long long)nbins < (1ull << 32);
    for (unsigned long long x0 = (unsigned long long)blockIdx.x * (8 * LNS_NT); x0 < N;
         x0 += (unsigned long long)gridDim.x * (8 * LNS_NT)) {
        int v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const unsigned long long x = x0 + (unsigned)u * LNS_NT + threadIdx.x;
            v[u] = x < N ? __ldcg(&A[x]) : 0;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            int b = -1;
            if (v[u] >= 1) {
                const uint32_t t = (uint32_t)(min(v[u], vmax) - 1);
                b = narrow ? (int)(t * (uint32_t)nbins / (uint32_t)vmax)
                           : (int)((unsigned long long)t * (unsigned long long)nbins / (unsigned long long)vmax);
            }
            const unsigned grp = __match_any_sync(0xffffffffu, b);
            if (b >= 0 && (int)(threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&lh[b], (uint32_t)__popc(grp));
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += blockDim.x)
        if (lh[b]) atomicAdd(&hist[b], (unsigned long long)lh[b]);
}

// The values behind an extraction threshold: those in (vmax / 2, vmax] in
// THR_BINS bins of `width` values, and the maximum of all.  vmax bounds the
// map (*vmax_dev where it is given).  The values of a map below half its
// maximum are nearly all of them and never reach the threshold, so a warp
// without a higher one only compares.
__device__ __forceinline__ int thr_width(int vmax) { return max(1, ((vmax + 1) / 2 + THR_BINS - 1) / THR_BINS); }

__global__ void __launch_bounds__(LNS_NT) k_lns_tail(const int32_t *A, uint32_t N, int vmax, const int *vmax_dev,
                                                     uint32_t *hist, int *top)
{
    __shared__ uint32_t lh[THR_BINS];
    for (int b = threadIdx.x; b < THR_BINS; b += LNS_NT) lh[b] = 0;
    if (vmax_dev) vmax = max(1, __ldcg(vmax_dev));
    __syncthreads();
    const int floor = vmax / 2, width = thr_width(vmax);
    int m = INT_MIN;
    for (unsigned long long x0 = (unsigned long long)blockIdx.x * (8 * LNS_NT); x0 < N;
         x0 += (unsigned long long)gridDim.x * (8 * LNS_NT)) {
        int v[8], w = INT_MIN;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const unsigned long long x = x0 + (unsigned)u * LNS_NT + threadIdx.x;
            v[u] = x < N ? __ldcg(&A[x]) : INT_MIN;
            w = max(w, v[u]);
        }
        m = max(m, w);
        if (!__any_sync(0xffffffffu, w > floor)) continue;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            // the lanes that share the first one's bin add once: early in a
            // fill all gains are equal, later they spread over the bins
            const int b = v[u] > floor ? min((v[u] - floor - 1) / width, THR_BINS - 1) : -1;
            const unsigned in = __ballot_sync(0xffffffffu, b >= 0);
            if (!in) continue;
            const int lead = __ffs(in) - 1, b0 = __shfl_sync(0xffffffffu, b, lead);
            const unsigned same = __ballot_sync(0xffffffffu, b == b0);
            if ((int)(threadIdx.x & 31) == lead) atomicAdd(&lh[b0], (uint32_t)__popc(same));
            else if (b >= 0 && b != b0) atomicAdd(&lh[b], 1u);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < THR_BINS; b += LNS_NT)
        if (lh[b]) atomicAdd(&hist[b], lh[b]);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(top, m);
}

// the threshold: the least value of the lowest bin whose tail holds at most
// cap words, but at most the maximum (which more than cap words may have)
__global__ void __launch_bounds__(THR_BINS) k_lns_threshold(const uint32_t *hist, int vmax, const int *vmax_dev,
                                                            long long cap, RefreshInfo *info)
{
    __shared__ unsigned long long ws[THR_BINS / 32];
    __shared__ int first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (vmax_dev) vmax = max(1, *vmax_dev);
    if (threadIdx.x == 0) first = THR_BINS;
    // the bin's tail: a prefix sum from the highest bin down
    const int b = THR_BINS - 1 - (int)threadIdx.x;
    unsigned long long x = hist[b];
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    for (int w = 0; w < warp; w++) x += ws[w];
    if (x <= (unsigned long long)cap) atomicMin(&first, b);
    __syncthreads();
    if (threadIdx.x == 0) info->thr = max(1, min(vmax / 2 + 1 + first * thr_width(vmax), info->top));
}

// ordered compaction of {x : A[x] >= thr}: counts of chunks of EXT_CHUNK
// words, their prefix sums, then positions; thr_dev (may be null) replaces thr
__global__ void __launch_bounds__(LNS_NT) k_lns_count_ge(const int32_t *A, uint32_t N, int thr, const int *thr_dev,
                                                         uint32_t *bcount)
{
    if (thr_dev) thr = __ldcg(thr_dev);
    const uint32_t x0 = blockIdx.x * EXT_CHUNK;
    uint32_t c = 0;
#pragma unroll 8
    for (uint32_t k = threadIdx.x; k < EXT_CHUNK; k += LNS_NT) {
        const uint32_t x = x0 + k;
        if (x < N) c += __ldcg(&A[x]) >= thr;
    }
    __shared__ uint32_t red[LNS_NT / 32];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int w = 0; w < LNS_NT / 32; w++) s += red[w];
        bcount[blockIdx.x] = s;
    }
}

// bcount[] -> its exclusive prefix sums (one block; saturated), the total to
// *found
__global__ void __launch_bounds__(1024) k_lns_scan(uint32_t *bcount, uint32_t nb, unsigned long long *found, uint32_t *found32)
{
    __shared__ unsigned long long ws[32], run;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) run = 0;
    __syncthreads();
    for (uint32_t b0 = 0; b0 < nb; b0 += 1024) {
        const uint32_t b = b0 + threadIdx.x;
        const unsigned long long c = b < nb ? bcount[b] : 0;
        unsigned long long x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        unsigned long long before = run;
        for (int w = 0; w < warp; w++) before += ws[w];
        if (b < nb) bcount[b] = (uint32_t)min(before + x - c, 0xffffffffull);
        __syncthreads();
        if (threadIdx.x == 1023) run = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (found) *found = run;
        if (found32) *found32 = (uint32_t)min(run, 0xffffffffull);
    }
}

__global__ void __launch_bounds__(LNS_NT) k_lns_emit_ge(const int32_t *A, uint32_t N, int thr, const int *thr_dev,
                                                        const uint32_t *boff, uint32_t cap, uint32_t *oidx, int32_t *oval)
{
    constexpr uint32_t SPAN = EXT_CHUNK / (LNS_NT / 32);      // consecutive words of a warp
    if (thr_dev) thr = __ldcg(thr_dev);
    const uint32_t first = boff[blockIdx.x];
    if (first >= cap || (blockIdx.x + 1 < gridDim.x && boff[blockIdx.x + 1] == first)) return;
    __shared__ uint32_t wcount[LNS_NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t x0 = blockIdx.x * EXT_CHUNK + (uint32_t)warp * SPAN + (uint32_t)lane;
    uint32_t c = 0;
#pragma unroll 8
    for (uint32_t k = 0; k < SPAN; k += 32) c += x0 + k < N && __ldcg(&A[x0 + k]) >= thr;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wcount[warp] = c;
    __syncthreads();
    if (!c) return;
    uint32_t at = first;
    for (int w = 0; w < warp; w++) at += wcount[w];
    for (uint32_t k = 0; k < SPAN; k += 32) {
        const uint32_t x = x0 + k;
        const int32_t v = x < N ? __ldcg(&A[x]) : INT_MIN;
        const bool take = x < N && v >= thr;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        const uint32_t to = at + __popc(m & ((1u << lane) - 1));
        if (take && to < cap) { oidx[to] = x; oval[to] = v; }
        at += __popc(m);
    }
}

// decode a packed word from its index
__device__ __forceinline__ uint64_t lns_pack(uint32_t x, int q, int n)
{
    uint64_t pk = 0;
    for (int j = n - 1; j >= 0; j--) { pk |= (uint64_t)(x % (uint32_t)q) << (4 * j); x /= (uint32_t)q; }
    return pk;
}

struct BallGeom {
    int q, n, R;
    uint32_t pw[COV_MAXN];
    const uint64_t *items;
    const uint8_t *last;
    uint32_t ngroups;
};

// The words of ball group `it` of the ball around base (packed pc): calls
// f(word) for each (one word, or the q-1 values of the group's last position).
template <class F>
__device__ __forceinline__ void ball_group(const BallGeom &b, uint32_t it, uint32_t base, uint64_t pc, F f)
{
    uint64_t sp = b.items[it];
    int off = (int)base;
    while (sp) {
        const int j = (__ffsll((long long)sp) - 1) >> 2;
        const int dig = (int)((sp >> (4 * j)) & 15u) - 1;
        sp &= ~(15ull << (4 * j));
        const int cj = cov_nib(pc, j);
        off += (dig + (dig >= cj) - cj) * (int)b.pw[j];
    }
    const int lj = b.last[it];
    if (lj == 0xff) {
        f((uint32_t)off);
    } else {
        const int step = (int)b.pw[lj], cj = cov_nib(pc, lj);
        int o2 = off - cj * step;
        for (int v = 0; v < b.q; v++, o2 += step)
            if (v != cj) f((uint32_t)o2);
    }
}

// One CTA per listed word: #{y in its ball : cnt[y] == target} (the
// independent exact counts of many words at once).
__global__ void k_lns_gather(const uint16_t *cnt, const uint32_t *idx, int k, BallGeom b, int target, int32_t *out)
{
    const int i = blockIdx.x;
    if (i >= k) return;
    const uint32_t base = idx[i];
    const uint64_t pc = lns_pack(base, b.q, b.n);
    int c = 0;
    for (uint32_t it = threadIdx.x; it < b.ngroups; it += blockDim.x)
        ball_group(b, it, base, pc, [&](uint32_t w) { c += __ldcg(&cnt[w]) == target; });
    __shared__ int red[32];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int w = 0; w < (int)(blockDim.x + 31) / 32; w++) s += red[w];
        out[i] = s;
    }
}

__global__ void k_lns_read(const int32_t *A, const uint32_t *idx, int k, int32_t *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < k) out[i] = A[idx[i]];
}

__global__ void k_lns_zero(const uint16_t *cnt, uint32_t N, int target, unsigned long long *out)
{
    unsigned long long c = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x)
        c += cnt[x] == target;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ------------------------------------------------- uncovered-word masks ----
// um[p]: bit y set iff the count of word p * blk + y is target.  A block of words
// (the blk = q^nb that share their high digits) is staged through shared
// memory, so that the counts are read once in order.
__global__ void __launch_bounds__(LNS_NT) k_lns_masks(const uint16_t *__restrict__ cnt, uint32_t nblk, int blk,
                                                      int target, uint64_t *__restrict__ um)
{
    __shared__ uint8_t z[LNS_NT * 64];
    const uint32_t p0 = blockIdx.x * LNS_NT;
    const uint32_t np = min((uint32_t)LNS_NT, nblk - p0);
    const uint16_t *c = cnt + (size_t)p0 * blk;
#pragma unroll 8
    for (uint32_t k = threadIdx.x; k < np * (uint32_t)blk; k += LNS_NT) z[k] = (int)__ldcg(&c[k]) == target;
    __syncthreads();
    if (threadIdx.x < np) {
        uint64_t m = 0;
        for (int y = 0; y < blk; y++) m |= (uint64_t)z[threadIdx.x * blk + y] << y;
        um[p0 + threadIdx.x] = m;
    }
}

// The words of um (all), or those that um_map has and um has not, into note in
// any order; um_map becomes um.  all < 0: none are noted.
__global__ void __launch_bounds__(LNS_NT) k_lns_note(const uint64_t *__restrict__ um, uint64_t *um_map, uint32_t nblk,
                                                     uint32_t blk, int all, uint32_t *note, uint32_t *noted)
{
    const uint32_t p = blockIdx.x * LNS_NT + threadIdx.x;
    uint64_t m = 0;
    if (p < nblk) {
        const uint64_t u = um[p];
        m = all > 0 ? u : all == 0 ? um_map[p] & ~u : 0;
        um_map[p] = u;
    }
    const uint32_t c = (uint32_t)__popcll(m);
    uint32_t at = c;
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    const uint32_t sum = __shfl_sync(0xffffffffu, at, 31);
    uint32_t base = 0;
    if (sum && lane == 0) base = atomicAdd(noted, sum);
    at += __shfl_sync(0xffffffffu, base, 0) - c;
    for (; m; m &= m - 1, at++)
        if (at < NOTE_CAP) note[at] = p * blk + (uint32_t)(__ffsll((long long)m) - 1);
}

// R = 0: the map is the marked words themselves
__global__ void k_lns_mask_words(const uint64_t *um, uint32_t N, uint32_t blk, int32_t *out)
{
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < N; x += gridDim.x * blockDim.x) {
        const uint32_t z = x / blk;
        out[x] = (int32_t)((um[z] >> (x - z * blk)) & 1u);
    }
}

// -------------------------------------------------------- lists of balls ----
// sgn over the balls of k listed words at once; the saturating updates of one
// sign commute, so the counts are those of one word after another.  *delta
// receives the change of the number of uncovered words.
__global__ void __launch_bounds__(LNS_NT) k_lns_apply(uint16_t *cnt, BallGeom b, const uint32_t *list, int k, int sgn,
                                                      uint32_t per, unsigned long long *delta)
{
    long long c = 0;
    const unsigned long long total = (unsigned long long)k * per;
    for (unsigned long long job = blockIdx.x; job < total; job += gridDim.x) {
        const uint32_t base = list[job / per];
        const uint32_t it = (uint32_t)(job % per) * LNS_NT + threadIdx.x;
        if (it >= b.ngroups) continue;
        const uint64_t pc = lns_pack(base, b.q, b.n);
        ball_group(b, it, base, pc, [&](uint32_t w) {
            unsigned short *p = reinterpret_cast<unsigned short *>(cnt) + w;
            unsigned short v = __ldcg(p);
            for (;;) {                                   // ends: a failed swap means another ball's succeeded
                if (v == (sgn > 0 ? 65535 : 0)) break;
                const unsigned short old = atomicCAS(p, v, (unsigned short)(v + sgn));
                if (old == v) {
                    if (sgn > 0) c -= v == 0;            // newly covered
                    else c += v == 1;                    // newly uncovered
                    break;
                }
                v = old;
            }
        });
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(delta, (unsigned long long)c);
}

// --------------------------------------------------------------- the greedy ----
struct GreedyArgs {
    uint16_t *cnt;
    uint64_t *um;
    BallGeom b, whole;             // the ball on the n - nb high digits (b.n of them), and on all
    const uint64_t *lowball;
    int nb, blk;
    uint64_t full;                 // the blk bits of a block
    const uint32_t *cand;          // candidates (increasing positions) and their exact gains
    const int32_t *bound;
    const RefreshInfo *info;
    uint32_t cand_cap;
    int room;                      // words still to place
    int eval_cap;                  // exact counts since the last placement after which a
                                   // fresh map is cheaper (the host refreshes)
    long long max_steps;           // bound on the steps of the launch
    int team, nteam;               // CTAs that count one candidate together; candidates at once
    int own;                       // most candidates of one CTA
    unsigned long long *nom;       // [2 * G]
    uint32_t *acc;                 // [3 * (GREEDY_MAXG + 1)]
    unsigned *bar;                 // arrivals at the grid barrier (cleared by the host)
    unsigned long long wait_ns;    // longest wait at a barrier
    uint32_t *list;
    SeqState *st;
};

// key of a candidate: larger bound first, then the lower position; 0: none
__device__ __forceinline__ unsigned long long cand_key(int32_t bound, int pos)
{
    return ((unsigned long long)(uint32_t)(bound + 0x40000000) << 32) | (uint32_t)(0x7fffffff - pos);
}
__device__ __forceinline__ int key_pos(unsigned long long k) { return 0x7fffffff - (int)(uint32_t)k; }
__device__ __forceinline__ int key_bound(unsigned long long k) { return (int)(uint32_t)(k >> 32) - 0x40000000; }

__device__ __forceinline__ unsigned long long warp_max64(unsigned long long k)
{
    for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
    return k;
}

// Greedy placement over the whole GPU, one CTA per SM.  CTA c owns the
// candidates p = c mod G, their bounds in its shared memory.  A step:
//   nominate: every CTA publishes the best key among its current bounds and
//     the best among its stale ones; the grid meets;
//   act: every CTA reads all keys and takes the same decision.  The best of
//     all is current: its ball is placed, and every bound becomes stale.  Else
//     the nteam best stale nominees above the best current one are counted
//     exactly, each by a team of CTAs; the grid meets.
// A word is placed only when its exact gain is at least every bound, so it is
// the word that counting one bound at a time would place.
//
// A count reads one mask per q^nb words instead of a counter per word (53,719
// gathers for 182,791 at q7 n9 R4, from 6.6 MB instead of 81 MB), and a step
// costs its two grid barriers and some six dependent trips to L2 whatever the
// number of candidates counted: 11 us for 25 candidates at 6^9, against 15 us
// for one on a cluster of 8 CTAs.  The fill of 6^9 (651 words) spends some 28
// ms here where the cluster took 247.
__global__ void __launch_bounds__(GREEDY_NT) k_lns_greedy(GreedyArgs a)
{
    extern __shared__ int gr_own[];                // [own] bounds, [own] epochs at which they were exact
    __shared__ unsigned long long s_stale[GREEDY_MAXG], s_team[GREEDY_MAXG], s_w[2][GREEDY_NT / 32];
    __shared__ unsigned long long s_kf, s_ks;
    __shared__ uint64_t s_low[8];
    __shared__ uint64_t s_pc, s_pw;                // the word's high digits, and all of them
    __shared__ unsigned s_sum[GREEDY_NT / 32];
    __shared__ int s_rank, s_count;
    const int G = (int)gridDim.x, me = (int)blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int *const sb = gr_own, *const sf = gr_own + a.own;
    const int ncand = (int)min(a.info->found, a.cand_cap);
    const int thr = a.info->thr;
    const int mine = ncand > me ? (ncand - me + G - 1) / G : 0;
    for (int i = threadIdx.x; i < mine; i += GREEDY_NT) { sb[i] = a.bound[me + i * G]; sf[i] = 1; }
    long long uncov = a.st->uncov, evals = 0, steps = 0;
    int epoch = 1, placed = 0, since = 0, status = SEQ_REFRESH, best = 0, buf = 0;
    unsigned met = 0;
    bool ok = ncand > 0;
    __syncthreads();
    while (ok) {
        // ---- nominate
        unsigned long long kf = 0, ks = 0;
        for (int i = threadIdx.x; i < mine; i += GREEDY_NT) {
            const unsigned long long k = cand_key(sb[i], me + i * G);
            if (sf[i] == epoch) kf = max(kf, k);
            else ks = max(ks, k);
        }
        kf = warp_max64(kf);
        ks = warp_max64(ks);
        if (lane == 0) { s_w[0][warp] = kf; s_w[1][warp] = ks; }
        __syncthreads();
        if (warp == 0) {
            kf = warp_max64(lane < GREEDY_NT / 32 ? s_w[0][lane] : 0);
            ks = warp_max64(lane < GREEDY_NT / 32 ? s_w[1][lane] : 0);
            if (lane == 0) { __stcg(&a.nom[me], kf); __stcg(&a.nom[G + me], ks); }
        }
        if (!(ok = cov_grid_meet(a.bar, ++met * (unsigned)G, a.wait_ns))) break;
        // ---- the decision, the same in every CTA
        kf = ks = 0;
        for (int t = threadIdx.x; t < G; t += GREEDY_NT) {
            kf = max(kf, __ldcg(&a.nom[t]));
            const unsigned long long s = __ldcg(&a.nom[G + t]);
            s_stale[t] = s;
            ks = max(ks, s);
        }
        kf = warp_max64(kf);
        ks = warp_max64(ks);
        if (lane == 0) { s_w[0][warp] = kf; s_w[1][warp] = ks; }
        __syncthreads();
        if (warp == 0) {
            kf = warp_max64(lane < GREEDY_NT / 32 ? s_w[0][lane] : 0);
            ks = warp_max64(lane < GREEDY_NT / 32 ? s_w[1][lane] : 0);
            if (lane == 0) { s_kf = kf; s_ks = ks; s_rank = -1; s_count = 0; }
        }
        __syncthreads();
        kf = s_kf;
        ks = s_ks;
        const unsigned long long top = max(kf, ks);
        const bool fresh = kf > ks;
        best = top ? key_bound(top) : 0;
        int stop = -1;
        if (uncov <= 0) stop = SEQ_COVERED;
        else if (placed >= a.room) stop = SEQ_TARGET;
        else if (++steps > a.max_steps) stop = SEQ_GUARD;
        // below the threshold a word outside the candidates could tie or beat
        // the best: the host refreshes the bounds (and stops when the fresh
        // map has no positive gain)
        else if (!top || best < thr) stop = SEQ_REFRESH;
        // so many bounds went stale that a fresh map is cheaper
        else if (!fresh && since >= a.eval_cap) stop = SEQ_REFRESH;
        if (stop >= 0) { status = stop; break; }
        uint32_t *const acc = a.acc + buf * (GREEDY_MAXG + 1);
        const int next = buf == 2 ? 0 : buf + 1;
        if (me == 0)               // last read two steps ago, next written in the next step
            for (int t = threadIdx.x; t <= a.nteam; t += GREEDY_NT) __stcg(&a.acc[next * (GREEDY_MAXG + 1) + t], 0u);
        int pos = -1, share = me, shares = G;
        if (fresh) {
            pos = key_pos(top);
        } else {
            // the nominees to count: the nteam best stale keys above the best
            // current one, each with its own team
            for (int t = threadIdx.x; t < G; t += GREEDY_NT) {
                const unsigned long long k = s_stale[t];
                if (k <= kf) continue;
                int rank = 0;
                for (int u = 0; u < G; u++) rank += s_stale[u] > k;
                if (rank < a.nteam) {
                    s_team[rank] = k;
                    if (t == me) s_rank = rank;
                    atomicAdd(&s_count, 1);
                }
            }
            __syncthreads();
            const int team = me / a.team;
            share = me - team * a.team;
            shares = a.team;
            if (team < s_count) pos = key_pos(s_team[team]);
        }
        unsigned c = 0;
        if (pos >= 0) {
            const uint32_t word = a.cand[pos];
            const uint32_t pre = word / (uint32_t)a.blk, low = word - pre * (uint32_t)a.blk;
            if (warp == 0) {
                uint32_t d = 0;
                if (lane < a.b.n) d = (pre / a.b.pw[lane]) % (uint32_t)a.b.q;
                const uint32_t lo = __reduce_or_sync(0xffffffffu, lane < 8 ? d << (4 * lane) : 0u);
                const uint32_t hi = __reduce_or_sync(0xffffffffu, lane >= 8 && lane < 16 ? d << (4 * (lane - 8)) : 0u);
                if (lane == 0) {
                    s_pc = ((uint64_t)hi << 32) | lo;
                    s_pw = s_pc;
                    for (uint32_t j = (uint32_t)a.whole.n, y = low; j-- > (uint32_t)a.b.n; y /= (uint32_t)a.b.q)
                        s_pw |= (uint64_t)(y % (uint32_t)a.b.q) << (4 * j);
                }
            } else if (warp == 1 && lane <= a.nb) {
                s_low[lane] = a.lowball[low * (uint32_t)(a.nb + 1) + (uint32_t)lane];
            }
            __syncthreads();
            const uint64_t pc = s_pc;
            const int R = (int)a.b.R;
            for (uint32_t it = (uint32_t)share * GREEDY_NT + threadIdx.x; it < a.b.ngroups;
                 it += (uint32_t)shares * GREEDY_NT) {
                const int r = __popcll(cov_spread(a.b.items[it])) + (a.b.last[it] != 0xff);
                const uint64_t m = R - r >= a.nb ? a.full : s_low[R - r];
                // each block of the ball is this thread's alone
                ball_group(a.b, it, pre, pc, [&](uint32_t p) {
                    const uint64_t u = __ldcg(&a.um[p]);
                    c += (unsigned)__popcll(u & m);
                    if (fresh && (u & m)) __stcg(&a.um[p], u & ~m);
                });
            }
            if (fresh) {
                // the counters, a word at a time (a block at a time they are a
                // chain of up to 64 dependent accesses: 130 us a placement)
                for (uint32_t it = (uint32_t)me * GREEDY_NT + threadIdx.x; it < a.whole.ngroups;
                     it += (uint32_t)G * GREEDY_NT)
                    ball_group(a.whole, it, word, s_pw, [&](uint32_t w) {
                        const uint16_t v = __ldcg(&a.cnt[w]);
                        if (v != 65535u) __stcg(&a.cnt[w], (uint16_t)(v + 1));
                    });
            }
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) s_sum[warp] = c;
            __syncthreads();
            if (threadIdx.x == 0) {
                unsigned t = 0;
                for (int w = 0; w < GREEDY_NT / 32; w++) t += s_sum[w];
                if (t) atomicAdd(&acc[fresh ? 0 : me / a.team], t);
            }
        }
        if (!(ok = cov_grid_meet(a.bar, ++met * (unsigned)G, a.wait_ns))) break;
        if (fresh) {
            if (threadIdx.x == 0 && me == 0) a.list[placed] = a.cand[pos];
            if (threadIdx.x == 0 && pos % G == me) sb[pos / G] = 0;      // a codeword now: its ball is covered
            uncov -= (long long)__ldcg(&acc[0]);
            placed++;
            epoch++;
            since = 0;
        } else {
            if (threadIdx.x == 0 && s_rank >= 0) {
                const int i = key_pos(s_stale[me]) / G;
                sb[i] = (int)__ldcg(&acc[s_rank]);
                sf[i] = epoch;
            }
            since += s_count;
            evals += s_count;
        }
        buf = next;
        __syncthreads();
    }
    if (me == 0 && threadIdx.x == 0) {
        a.st->uncov = uncov;
        a.st->evals = evals;
        a.st->placed = placed;
        a.st->status = !ok && ncand > 0 ? SEQ_GUARD : status;
        a.st->best = max(best, thr);
    }
}

// ------------------------------------------------------------ the peel ----
struct SeqArgs {
    uint16_t *cnt;
    BallGeom b;
    long long max_steps;           // bound on the steps of one launch
    uint32_t *list;                // the codewords in order
    int nlist;
    uint8_t *flag;
    SeqState *st;
};

struct SeqShared {
    long long sum;                 // ball count / crossings over the cluster
    int act;                       // the leader's decision
    uint32_t word;
};

// a ball walked by the whole cluster: count (op 0: cnt == 1) or subtract (op
// 1; returns the words that became uncovered).  All words of one ball are
// distinct.
__device__ __forceinline__ long long cluster_ball(const SeqArgs &a, uint32_t base, int op, int rank)
{
    const uint64_t pc = lns_pack(base, a.b.q, a.b.n);
    long long c = 0;
    for (uint32_t it = (uint32_t)rank * SEQ_NT + threadIdx.x; it < a.b.ngroups; it += SEQ_CL * SEQ_NT) {
        ball_group(a.b, it, base, pc, [&](uint32_t w) {
            const uint32_t v = __ldcg(&a.cnt[w]);
            c += v == 1u;
            if (op && v != 0u) __stcg(&a.cnt[w], (uint16_t)(v - 1));
        });
    }
    return c;
}

// reduce a per-thread value into the leader CTA's shared sum
__device__ __forceinline__ void cluster_add(long long v, SeqShared *lead)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd((unsigned long long *)&lead->sum, (unsigned long long)v);
}

enum { ACT_STOP = 0, ACT_EVAL, ACT_REMOVE, ACT_NEXT };

__global__ void __cluster_dims__(SEQ_CL, 1, 1) __launch_bounds__(SEQ_NT) k_lns_peel(SeqArgs a)
{
    __shared__ SeqShared sh;
    __shared__ long long s_uncov, s_evals, s_steps;
    __shared__ int s_removed, s_i;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    SeqShared *lead = cl.map_shared_rank(&sh, 0);
    if (threadIdx.x == 0) {
        sh.sum = 0; sh.act = ACT_NEXT; sh.word = 0;
        if (rank == 0) { s_uncov = a.st->uncov; s_evals = 0; s_steps = 0; s_removed = 0; s_i = 0; }
    }
    __syncthreads();
    cl.sync();
    for (;;) {
        // every CTA has read the previous step's decision before the leader
        // writes the next one
        cl.sync();
        if (rank == 0 && threadIdx.x == 0) {
            if (s_i >= a.nlist || ++s_steps > a.max_steps) {
                sh.act = ACT_STOP;
                a.st->status = s_i >= a.nlist ? SEQ_DONE : SEQ_GUARD;
            } else {
                sh.act = ACT_EVAL;
                sh.word = a.list[s_i];
            }
            sh.sum = 0;
        }
        cl.sync();
        const uint32_t word = lead->word;
        if (lead->act == ACT_STOP) break;
        // the exact loss: ball words covered only once
        cluster_add(cluster_ball(a, word, 0, rank), lead);
        cl.sync();
        if (rank == 0 && threadIdx.x == 0) {
            s_evals++;
            sh.act = sh.sum == 0 ? ACT_REMOVE : ACT_NEXT;    // remove it if it covers nothing alone
            if (sh.act == ACT_NEXT) s_i++;
            sh.sum = 0;
        }
        cl.sync();
        if (lead->act != ACT_REMOVE) continue;
        cluster_add(cluster_ball(a, word, 1, rank), lead);
        cl.sync();
        if (rank == 0 && threadIdx.x == 0) {
            s_uncov += sh.sum;
            sh.sum = 0;
            a.flag[s_i] = 1;
            s_removed++;
            s_i++;
        }
        cl.sync();
    }
    if (rank == 0 && threadIdx.x == 0) {
        a.st->uncov = s_uncov;
        a.st->evals = s_evals;
        a.st->placed = 0;
        a.st->removed = s_removed;
    }
    // no CTA may leave while another can still reach the leader's shared memory
    cl.sync();
}

int grid_of(uint32_t N)
{
    return (int)std::min<uint32_t>((N + LNS_NT - 1) / LNS_NT, (uint32_t)std::max(1, cov_sm_count()) * 8);
}

CovDeviceFlags g_map_attr;      // shared-memory opt-in of the map kernels, per device

void map_kernels(int q, int layers, MapLow *low, MapHigh *high)
{
    switch (map_slots(layers)) {
    case 3: map_kernels_3(q, low, high); break;
    case 5: map_kernels_5(q, low, high); break;
    case 7: map_kernels_7(q, low, high); break;
    default: map_kernels_9(q, low, high); break;
    }
}

int map_attrs()
{
    int dev = 0;
    if (g_map_attr.done(dev)) return 0;
    for (int q = 2; q <= 11; q++)
        for (int layers : {3, 5, 7, 9}) {
            MapLow low;
            MapHigh high;
            map_kernels(q, layers, &low, &high);
            CK(cudaFuncSetAttribute((const void *)low, cudaFuncAttributeMaxDynamicSharedMemorySize, MAP_SMEM_MAX));
            CK(cudaFuncSetAttribute((const void *)high, cudaFuncAttributeMaxDynamicSharedMemorySize, MAP_SMEM_MAX));
        }
    g_map_attr.set(dev);
    return 0;
}

// The layered transform of the marked words (masks um) or of the word counts
// A0, result to out (int32 map) or cnt16.
int lns_transform(cov_lns *h, const int32_t *A0, int32_t *out, uint16_t *cnt16)
{
    int rc = map_attrs();
    if (rc) return rc;
    const int q = h->q, n = h->n, R = h->R, sms = std::max(1, cov_sm_count());
    MapLow low;
    MapHigh high;
    MapGeom g;
    memset(&g, 0, sizeof g);
    g.q = q; g.n = n; g.R = R;
    g.T = (uint32_t)bt_ipow(q, h->kl);
    g.Tp = map_cols(q, h->kl);
    g.out = out; g.cnt16 = cnt16;
    auto grid_for = [&](uint32_t tiles, size_t smem) {
        const uint32_t per_sm = (uint32_t)std::max<size_t>(1, std::min<size_t>(8, 225 * 1024 / (smem + 1024)));
        return std::min(tiles, (uint32_t)sms * per_sm);
    };
    // strip sweep i over `tiles` low tiles
    auto strips = [&](int i, int j0, uint32_t tiles, const int32_t *from, int32_t *to, int slots) {
        const int gsz = h->gs[i];
        const uint32_t s = (uint32_t)bt_ipow(q, j0 - h->kl) * g.Tp, rows = (uint32_t)bt_ipow(q, gsz);
        const size_t per = (size_t)rows * h->slots[i] * 4;
        int lw = 3;
        while (per * ((size_t)2 << lw) <= MAP_SMEM_HIGH && (1u << lw) < s && lw < 6) lw++;
        const uint32_t nt = tiles / (uint32_t)bt_ipow(q, j0 + gsz - h->kl) * ((s + (1u << lw) - 1) >> lw);
        map_kernels(q, h->slots[i], &low, &high);
        high<<<grid_for(nt, per << lw), MAP_HIGH_NT, per << lw>>>(g, j0, gsz, lw, s, nt, from, to, slots);
        CK(cudaGetLastError());
        return 0;
    };
    const int lslots = h->low_slots(R);
    const size_t lsm = map_low_smem(q, lslots, h->kl, h->nb, h->blk);
    const uint32_t part_tiles = h->N / h->parts / g.T;
    for (uint32_t p = 0; p < h->parts; p += h->at_once) {
        const uint32_t t0 = p * part_tiles, tiles = std::min(h->at_once, h->parts - p) * part_tiles;
        map_kernels(q, lslots, &low, &high);
        low<<<grid_for(tiles, lsm), MAP_LOW_NT, lsm>>>(g, h->kl, h->nb, h->blk, A0 ? nullptr : h->um, h->lowball, A0, t0,
                                                       tiles, h->map_scratch, h->ng ? h->slots[0] : 0);
        CK(cudaGetLastError());
        int j0 = h->kl;
        int32_t *from = h->map_scratch, *other = h->map_scratch + h->scratch_ints;
        for (int i = 0; i < h->ng && (i == 0 || i < h->ng - 1); i++) {
            const bool last = h->ng >= 2 && i == h->ng - 2;
            int32_t *to = last ? h->map_whole + (size_t)t0 * g.Tp * h->slots[h->ng - 1] : other;
            rc = strips(i, j0, tiles, from, to, i + 1 < h->ng ? h->slots[i + 1] : 0);
            if (rc) return rc;
            other = from;
            from = to;
            j0 += h->gs[i];
        }
    }
    if (h->ng >= 2) return strips(h->ng - 1, n - h->gs[h->ng - 1], h->N / g.T, h->map_whole, nullptr, 0);
    return 0;
}

// masks of the words whose count is target
int lns_masks(cov_lns *h, int target)
{
    const uint32_t nblk = h->N / h->blk;
    k_lns_masks<<<(nblk + LNS_NT - 1) / LNS_NT, LNS_NT>>>(h->cnt, nblk, (int)h->blk, target, h->um);
    CK(cudaGetLastError());
    return 0;
}

// the map of the words whose masks are in um
int lns_map_of_masks(cov_lns *h)
{
    if (h->R > 0) return lns_transform(h, nullptr, h->map, nullptr);
    k_lns_mask_words<<<grid_of(h->N), LNS_NT>>>(h->um, h->N, h->blk, h->map);
    CK(cudaGetLastError());
    return 0;
}

// The greedy's map of the uncovered words (masks um, `left` of them).  Few
// uncovered words are counted by tiles from their list; few words covered
// since the last map (`gone` of them; < 0: there is no last map) are counted
// off it; else the transform of the masks, one launch less (spaces below a
// million words gain nothing: 17 to 90 ms fills of 6^6 to 7^7 with and
// without).  Map at 7^9: 0.92 ms by transform, 0.07 to 0.25 by
// tiles of 10 to 3000 words.  Six rounds at 7^9 48 -> 29 ms (25 with fewer
// exact counts before a refresh), the fill of 6^9 71 -> 65.
// *tiled: the map came from tiles.
int lns_greedy_map(cov_lns *h, long long left, long long gone, bool *tiled)
{
    const int sms = std::max(1, cov_sm_count());
    const double all_ps = left <= NOTE_CAP ? bt_count_ps(h->q, h->n, h->R, left, sms) + 0.6 * h->N : 1e300;
    const double off_ps = gone >= 0 && gone <= NOTE_CAP ? bt_count_ps(h->q, h->n, h->R, gone, sms) + 1.2 * h->N : 1e300;
    *tiled = false;
    if (h->R == 0 || h->N <= MAP_TILES_N) return lns_map_of_masks(h);
    const bool tiles = bt_transform_ps(h->R) * h->N - std::min(all_ps, off_ps) > MAP_PS_LAUNCH;
    const int how = !tiles ? -1 : all_ps <= off_ps ? 1 : 0;
    const uint32_t nblk = h->N / h->blk;
    CK(cudaMemsetAsync(&h->info->noted, 0, 4));
    k_lns_note<<<(nblk + LNS_NT - 1) / LNS_NT, LNS_NT>>>(h->um, h->um_map, nblk, h->blk, how, h->note, &h->info->noted);
    CK(cudaGetLastError());
    if (how < 0) return lns_map_of_masks(h);
    *tiled = true;
    return cov_count_words_map(h->q, h->n, h->R, h->note, (int)(how ? left : gone), h->map, !how,
                               (uint2 *)(h->note + NOTE_CAP), nullptr);
}

int lns_scratch(cov_lns *h, size_t bytes)
{
    if (bytes <= h->scratch_bytes) return 0;
    if (h->scratch) cudaFree(h->scratch);
    h->scratch = nullptr;
    h->scratch_bytes = 0;
    if (cudaMalloc(&h->scratch, bytes) != cudaSuccess) { cudaGetLastError(); return COV_ENOMEM; }
    h->scratch_bytes = bytes;
    return 0;
}

BallGeom ball_geom(const cov_lns *h)
{
    BallGeom b;
    memset(&b, 0, sizeof b);
    b.q = h->q; b.n = h->n; b.R = h->R;
    for (int j = 0; j < h->n; j++) b.pw[j] = h->pw[j];
    b.items = h->ball; b.last = h->ball_last; b.ngroups = h->ngroups;
    return b;
}

// the ball on the high digits, whose words are the mask blocks
BallGeom block_geom(const cov_lns *h)
{
    BallGeom b;
    memset(&b, 0, sizeof b);
    b.q = h->q; b.n = h->n - h->nb; b.R = h->R;
    for (int j = 0; j < b.n; j++) b.pw[j] = h->pw[j] / h->blk;
    b.items = h->pball; b.last = h->pball_last; b.ngroups = h->npgroups;
    return b;
}

long long count_eq(cov_lns *h, int target)
{
    if (cudaMemset(h->d_red, 0, 8) != cudaSuccess) return -1;
    k_lns_zero<<<grid_of(h->N), LNS_NT>>>(h->cnt, h->N, target, h->d_red);
    unsigned long long z = 0;
    if (cudaMemcpy(&z, h->d_red, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    return (long long)z;
}

// room for a list of k words (and their flags) on the device
int list_room(cov_lns *h, int k)
{
    if (k > h->list_cap) {
        cudaFree(h->list);
        cudaFree(h->flag);
        h->list = nullptr;
        h->flag = nullptr;
        h->list_cap = 0;
        CK(cudaMalloc(&h->list, (size_t)k * 4));
        CK(cudaMalloc(&h->flag, (size_t)k));
        h->list_cap = k;
    }
    return 0;
}

// ordered extraction into device buffers (oidx, oval) of at most cap entries;
// thr_dev (may be null) replaces thr.  bcount: extract_blocks(h) words.
uint32_t extract_blocks(const cov_lns *h) { return (h->N + EXT_CHUNK - 1) / EXT_CHUNK; }

int extract_launch(cov_lns *h, int32_t thr, const int *thr_dev, int64_t cap, uint32_t *bcount, uint32_t *oidx,
                   int32_t *oval, unsigned long long *found, uint32_t *found32)
{
    const uint32_t nb = extract_blocks(h);
    k_lns_count_ge<<<nb, LNS_NT>>>(h->map, h->N, thr, thr_dev, bcount);
    k_lns_scan<<<1, 1024>>>(bcount, nb, found, found32);
    if (cap > 0)
        k_lns_emit_ge<<<nb, LNS_NT>>>(h->map, h->N, thr, thr_dev, bcount,
                                      (uint32_t)std::min<int64_t>(cap, 0xffffffffll), oidx, oval);
    CK(cudaGetLastError());
    return COV_OK;
}

// the greedy kernel's launch shape on the current device
int greedy_shape(cov_lns *h, GreedyArgs &a, int *G, size_t *smem)
{
    *G = std::min(std::max(1, cov_sm_count()), GREEDY_MAXG);
    a.own = (CAND_CAP + *G - 1) / *G;
    *smem = (size_t)a.own * 8;
    // a team's threads take about two groups each
    a.team = (int)std::min<uint32_t>((uint32_t)*G, std::max(1u, (h->npgroups + 2 * GREEDY_NT - 1) / (2 * GREEDY_NT)));
    a.nteam = *G / a.team;
    if (*smem > 48 * 1024) CK(cudaFuncSetAttribute(k_lns_greedy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem));
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lns_greedy, GREEDY_NT, *smem));
    return per_sm >= 1 ? COV_OK : COV_ENODEV;
}

}  // namespace

extern "C" {

int cov_lns_create(int32_t q, int32_t n, int32_t R, cov_lns **out)
{
    if (!out || q < 2 || q > 16 || n < 1 || n > 16 || R < 0 || R > LNS_MAXR) return COV_EINVAL;
    long long N = 1;
    for (int j = 0; j < n; j++) N *= q;
    if (N >= (1LL << 31)) return COV_ERANGE;
    if (R > n) R = n;
    int dev_count = 0;
    if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0) { cudaGetLastError(); return COV_ENODEV; }
    cov_lns *h = new cov_lns;
    h->q = q; h->n = n; h->R = R; h->N = (uint32_t)N;
    for (int j = 0; j < n; j++) { long long p = 1; for (int k = 0; k < n - 1 - j; k++) p *= q; h->pw[j] = (uint32_t)p; }
    std::vector<uint8_t> last;
    uint32_t gcum[COV_MAXN + 2];
    std::vector<uint64_t> items = bt_items_h(q, n, R, 0, gcum, last);
    h->ngroups = gcum[std::min(R, n)];
    // mask blocks: the ball groups on the high digits, and for each word of a
    // block the words of it within 0..nb
    while (h->nb < n && (long long)h->blk * q <= 64) { h->nb++; h->blk *= (uint32_t)q; }
    std::vector<uint8_t> plast;
    uint32_t pcum[COV_MAXN + 2];
    std::vector<uint64_t> pitems = bt_items_h(q, n - h->nb, R, 0, pcum, plast);
    h->npgroups = pcum[std::min(R, n - h->nb)];
    std::vector<uint64_t> low((size_t)h->blk * (h->nb + 1), 0);
    for (uint32_t x = 0; x < h->blk; x++)
        for (uint32_t y = 0; y < h->blk; y++) {
            int d = 0;
            for (uint32_t u = x, v = y, k = 0; k < (uint32_t)h->nb; k++, u /= q, v /= q) d += u % q != v % q;
            for (int sg = d; sg <= h->nb; sg++) low[(size_t)x * (h->nb + 1) + sg] |= 1ull << y;
        }
    map_plan(*h, q, n, R, h->N, h->nb, h->blk);
    bool ok = cudaMalloc(&h->cnt, (size_t)N * 2) == cudaSuccess &&
              cudaMalloc(&h->map, (size_t)N * 4) == cudaSuccess &&
              cudaMalloc(&h->ball, items.size() * 8) == cudaSuccess &&
              cudaMalloc(&h->ball_last, last.size()) == cudaSuccess &&
              cudaMalloc(&h->d_red, 64 * 8) == cudaSuccess &&
              cudaMalloc(&h->cand, (size_t)CAND_CAP * 4) == cudaSuccess &&
              cudaMalloc(&h->bound, (size_t)CAND_CAP * 4) == cudaSuccess &&
              cudaMalloc(&h->um, (size_t)(N / h->blk) * 8) == cudaSuccess &&
              cudaMalloc(&h->um_map, (size_t)(N / h->blk) * 8) == cudaSuccess &&
              cudaMalloc(&h->note, (size_t)NOTE_CAP * (4 + BT_REC_BYTES)) == cudaSuccess &&
              cudaMalloc(&h->pball, pitems.size() * 8) == cudaSuccess &&
              cudaMalloc(&h->pball_last, plast.size()) == cudaSuccess &&
              cudaMalloc(&h->lowball, low.size() * 8) == cudaSuccess &&
              cudaMalloc(&h->nom, sizeof(unsigned long long) * 2 * GREEDY_MAXG) == cudaSuccess &&
              cudaMalloc(&h->acc, 4 * (3 * (GREEDY_MAXG + 1) + 1)) == cudaSuccess &&
              cudaMalloc(&h->info, sizeof(RefreshInfo)) == cudaSuccess &&
              cudaMalloc(&h->seq, sizeof(SeqState)) == cudaSuccess;
    if (ok)
        ok = cudaMalloc(&h->map_scratch, (h->scratch_ints * (h->ng >= 3 ? 2 : 1) + h->counts_ints) * 4) == cudaSuccess;
    if (ok && h->whole_ints) ok = cudaMalloc(&h->map_whole, h->whole_ints * 4) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        cov_lns_destroy(h);
        return COV_ENOMEM;
    }
    if (cudaMemcpy(h->ball, items.data(), items.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->ball_last, last.data(), last.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->pball, pitems.data(), pitems.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->pball_last, plast.data(), plast.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->lowball, low.data(), low.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(h->cnt, 0, (size_t)N * 2) != cudaSuccess) {
        cov_lns_destroy(h);
        return -100;
    }
    *out = h;
    return COV_OK;
}

int cov_lns_destroy(cov_lns *h)
{
    if (!h) return COV_OK;
    cudaDeviceSynchronize();
    cudaFree(h->cnt); cudaFree(h->map); cudaFree(h->ball); cudaFree(h->ball_last); cudaFree(h->d_red);
    cudaFree(h->cand); cudaFree(h->bound); cudaFree(h->list); cudaFree(h->flag); cudaFree(h->seq);
    cudaFree(h->um); cudaFree(h->um_map); cudaFree(h->note); cudaFree(h->pball); cudaFree(h->pball_last); cudaFree(h->lowball); cudaFree(h->nom);
    cudaFree(h->acc); cudaFree(h->info); cudaFree(h->map_scratch); cudaFree(h->map_whole);
    cudaFree(h->scratch);
    delete h;
    return COV_OK;
}

int cov_lns_recount(cov_lns *h, const uint32_t *idx, int32_t m)
{
    if (!h || m < 0 || (m > 0 && !idx)) return COV_EINVAL;
    for (int i = 0; i < m; i++) if (idx[i] >= h->N) return COV_EINVAL;
    // the verifier's tiles while the code is sparse, else the transform of its
    // word counts
    if (bt_tiles_pay(h->q, h->n, h->R, m, std::max(1, cov_sm_count()))) {
        int rc = lns_scratch(h, (size_t)m * (4 + BT_REC_BYTES) + 8);
        if (rc) return rc;
        uint2 *rec = (uint2 *)h->scratch;
        uint32_t *d_i = (uint32_t *)((char *)h->scratch + (size_t)m * BT_REC_BYTES);
        if (m > 0) CK(cudaMemcpy(d_i, idx, (size_t)m * 4, cudaMemcpyHostToDevice));
        rc = cov_count_words(h->q, h->n, h->R, d_i, m, h->cnt, rec, nullptr);
        if (rc) return rc;
        CK(cudaDeviceSynchronize());
        return COV_OK;
    }
    int rc = lns_scratch(h, (size_t)m * 4);
    if (rc) return rc;
    // (in the handle's own memory: an allocation of 4 q^n bytes for the call
    // took 200 of the 508 us of 200,000 words at 7^8 R5, and could fail)
    int32_t *const a0 = h->ng >= 2 ? h->map_whole + h->counts_at : h->map_scratch + h->scratch_ints;
    CK(cudaMemsetAsync(a0, 0, (size_t)h->N * 4));
    CK(cudaMemcpy(h->scratch, idx, (size_t)m * 4, cudaMemcpyHostToDevice));
    k_lns_scatter<<<(m + 255) / 256, 256>>>(a0, (const uint32_t *)h->scratch, m);
    CK(cudaGetLastError());
    if (h->R == 0) k_lns_narrow<<<grid_of(h->N), LNS_NT>>>(a0, h->N, h->cnt);
    else rc = lns_transform(h, a0, nullptr, h->cnt);
    if (rc) return rc;
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
    return COV_OK;
}

int cov_lns_map(cov_lns *h, int32_t target)
{
    if (!h || target < 0) return COV_EINVAL;
    int rc = lns_masks(h, target);
    if (!rc) rc = lns_map_of_masks(h);
    if (rc) return rc;
    CK(cudaDeviceSynchronize());
    return COV_OK;
}

int cov_lns_map_max(cov_lns *h, int32_t *out)
{
    if (!h || !out) return COV_EINVAL;
    const int init = INT32_MIN;
    CK(cudaMemcpy(h->d_red, &init, 4, cudaMemcpyHostToDevice));
    k_lns_max<<<grid_of(h->N), LNS_NT>>>(h->map, h->N, (int *)h->d_red);
    CK(cudaGetLastError());
    CK(cudaMemcpy(out, h->d_red, 4, cudaMemcpyDeviceToHost));
    return COV_OK;
}

int cov_lns_map_hist(cov_lns *h, int32_t nbins, int32_t vmax, int64_t *hist)
{
    if (!h || !hist || nbins < 1 || nbins > LNS_HIST_MAX || vmax < 1) return COV_EINVAL;
    int rc = lns_scratch(h, (size_t)nbins * 8);
    if (rc) return rc;
    unsigned long long *d_h = (unsigned long long *)h->scratch;
    CK(cudaMemset(d_h, 0, (size_t)nbins * 8));
    k_lns_hist<<<grid_of(h->N), LNS_NT, (size_t)nbins * 4>>>(h->map, h->N, nbins, vmax, d_h);
    CK(cudaGetLastError());
    CK(cudaMemcpy(hist, d_h, (size_t)nbins * 8, cudaMemcpyDeviceToHost));
    return COV_OK;
}

int cov_lns_map_extract(cov_lns *h, int32_t thr, int64_t cap, uint32_t *idx, int32_t *val, int64_t *found)
{
    if (!h || cap < 0 || (cap > 0 && (!idx || !val)) || !found) return COV_EINVAL;
    const uint32_t nb = extract_blocks(h);
    // at most N entries are written
    const int64_t room = std::min<int64_t>(cap, (int64_t)h->N);
    const size_t cb = ((size_t)nb * 4 + 7) / 8 * 8;
    int rc = lns_scratch(h, cb + 8 + (size_t)room * 8);
    if (rc) return rc;
    uint32_t *bcount = (uint32_t *)h->scratch;
    unsigned long long *d_f = (unsigned long long *)((char *)h->scratch + cb), tot = 0;
    uint32_t *d_i = (uint32_t *)(d_f + 1);
    int32_t *d_v = (int32_t *)(d_i + room);
    rc = extract_launch(h, thr, nullptr, room, bcount, d_i, d_v, d_f, nullptr);
    if (rc) return rc;
    CK(cudaMemcpy(&tot, d_f, 8, cudaMemcpyDeviceToHost));
    *found = (int64_t)tot;
    const size_t k = (size_t)std::min<int64_t>(*found, room);
    if (k) {
        CK(cudaMemcpy(idx, d_i, k * 4, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(val, d_v, k * 4, cudaMemcpyDeviceToHost));
    }
    return COV_OK;
}

int cov_lns_map_read(cov_lns *h, const uint32_t *idx, int32_t k, int32_t *out)
{
    if (!h || k < 0 || (k > 0 && (!idx || !out))) return COV_EINVAL;
    if (k == 0) return COV_OK;
    for (int i = 0; i < k; i++) if (idx[i] >= h->N) return COV_EINVAL;
    int rc = lns_scratch(h, (size_t)k * 8);
    if (rc) return rc;
    uint32_t *d_i = (uint32_t *)h->scratch;
    int32_t *d_o = (int32_t *)(d_i + k);
    CK(cudaMemcpy(d_i, idx, (size_t)k * 4, cudaMemcpyHostToDevice));
    k_lns_read<<<(k + 255) / 256, 256>>>(h->map, d_i, k, d_o);
    CK(cudaGetLastError());
    CK(cudaMemcpy(out, d_o, (size_t)k * 4, cudaMemcpyDeviceToHost));
    return COV_OK;
}

int cov_lns_apply(cov_lns *h, const uint32_t *idx, int32_t k, int32_t sign, int64_t *uncovered)
{
    if (!h || k < 0 || (k > 0 && !idx) || (sign != 1 && sign != -1) || !uncovered) return COV_EINVAL;
    for (int i = 0; i < k; i++) if (idx[i] >= h->N) return COV_EINVAL;
    // the uncovered words before, and their change, in one counter
    CK(cudaMemsetAsync(h->d_red, 0, 8));
    k_lns_zero<<<grid_of(h->N), LNS_NT>>>(h->cnt, h->N, 0, h->d_red);
    CK(cudaGetLastError());
    if (k > 0) {
        int rc = list_room(h, k);
        if (rc) return rc;
        CK(cudaMemcpy(h->list, idx, (size_t)k * 4, cudaMemcpyHostToDevice));
        const uint32_t per = (h->ngroups + LNS_NT - 1) / LNS_NT;
        const int grid = (int)std::min<unsigned long long>((unsigned long long)k * per,
                                                           (unsigned long long)std::max(1, cov_sm_count()) * 8);
        k_lns_apply<<<grid, LNS_NT>>>(h->cnt, ball_geom(h), h->list, k, sign, per, h->d_red);
        CK(cudaGetLastError());
    }
    unsigned long long u = 0;
    CK(cudaMemcpy(&u, h->d_red, 8, cudaMemcpyDeviceToHost));
    *uncovered = (int64_t)u;
    return COV_OK;
}

int cov_lns_ball(cov_lns *h, const uint32_t *idx, int32_t k, int32_t op, int32_t arg, int32_t *out)
{
    if (!h || k < 0 || (k > 0 && !idx) || op < 0 || op > 1 || (op == 0 && k > 0 && !out)) return COV_EINVAL;
    if (k == 0) return COV_OK;
    for (int i = 0; i < k; i++) if (idx[i] >= h->N) return COV_EINVAL;
    if (op == 0) {
        int rc = lns_scratch(h, (size_t)k * 8);
        if (rc) return rc;
        uint32_t *d_i = (uint32_t *)h->scratch;
        int32_t *d_o = (int32_t *)(d_i + k);
        CK(cudaMemcpy(d_i, idx, (size_t)k * 4, cudaMemcpyHostToDevice));
        k_lns_gather<<<k, LNS_NT>>>(h->cnt, d_i, k, ball_geom(h), arg, d_o);
        CK(cudaGetLastError());
        CK(cudaMemcpy(out, d_o, (size_t)k * 4, cudaMemcpyDeviceToHost));
        return COV_OK;
    }
    int64_t unc = 0;
    return cov_lns_apply(h, idx, k, arg, &unc);
}

int cov_lns_peel(cov_lns *h, const uint32_t *idx, int32_t k, uint8_t *removed, int32_t *nremoved,
                 int64_t *uncovered)
{
    if (!h || k < 0 || (k > 0 && (!idx || !removed)) || !nremoved || !uncovered) return COV_EINVAL;
    for (int i = 0; i < k; i++) if (idx[i] >= h->N) return COV_EINVAL;
    SeqState st;
    memset(&st, 0, sizeof st);
    st.uncov = count_eq(h, 0);
    if (st.uncov < 0) return -100;
    *nremoved = 0;
    if (k > 0) {
        int rc = list_room(h, k);
        if (rc) return rc;
        CK(cudaMemcpy(h->list, idx, (size_t)k * 4, cudaMemcpyHostToDevice));
        CK(cudaMemset(h->flag, 0, (size_t)k));
        SeqArgs a;
        memset(&a, 0, sizeof a);
        a.cnt = h->cnt; a.b = ball_geom(h); a.st = h->seq;
        a.list = h->list; a.nlist = k; a.flag = h->flag;
        a.max_steps = 2LL * k + 2;
        CK(cudaMemcpy(h->seq, &st, sizeof st, cudaMemcpyHostToDevice));
        k_lns_peel<<<SEQ_CL, SEQ_NT>>>(a);
        CK(cudaGetLastError());
        CK(cudaMemcpy(&st, h->seq, sizeof st, cudaMemcpyDeviceToHost));
        if (st.status != SEQ_DONE) return COV_ETIMEOUT;
        CK(cudaMemcpy(removed, h->flag, (size_t)k, cudaMemcpyDeviceToHost));
        *nremoved = st.removed;
    }
    *uncovered = st.uncov;
    return COV_OK;
}

int cov_lns_greedy(cov_lns *h, int32_t room, int64_t cand_cap, uint32_t *placed, int32_t *nplaced,
                   int64_t *uncovered, int64_t *stats)
{
    if (!h || room < 0 || (room > 0 && !placed) || !nplaced || !uncovered) return COV_EINVAL;
    cand_cap = std::max<int64_t>(1, std::min<int64_t>(cand_cap > 0 ? cand_cap : CAND_CAP, CAND_CAP));
    int rc = list_room(h, room);
    if (rc) return rc;
    GreedyArgs a;
    memset(&a, 0, sizeof a);
    int G = 1;
    size_t smem = 0;
    rc = greedy_shape(h, a, &G, &smem);
    if (rc) return rc;
    const uint32_t xb = extract_blocks(h);
    rc = lns_scratch(h, THR_BINS * 4 + (size_t)xb * 4);
    if (rc) return rc;
    uint32_t *d_hist = (uint32_t *)h->scratch;
    uint32_t *bcount = (uint32_t *)(d_hist + THR_BINS);
    SeqState st;
    memset(&st, 0, sizeof st);
    st.uncov = count_eq(h, 0);
    if (st.uncov < 0) return -100;
    CK(cudaMemcpy(h->seq, &st, sizeof st, cudaMemcpyHostToDevice));
    // the uncovered words' masks, which the placements keep current
    if (room > 0 && st.uncov > 0) {
        rc = lns_masks(h, 0);
        if (rc) return rc;
    }
    a.cnt = h->cnt; a.um = h->um; a.b = block_geom(h); a.whole = ball_geom(h); a.lowball = h->lowball;
    a.nb = h->nb; a.blk = (int)h->blk;
    a.full = h->blk == 64 ? ~0ull : (1ull << h->blk) - 1;
    a.cand = h->cand; a.bound = h->bound; a.info = h->info; a.cand_cap = (uint32_t)cand_cap;
    a.nom = h->nom; a.acc = h->acc; a.bar = h->acc + 3 * (GREEDY_MAXG + 1);
    a.wait_ns = 2000000000ull;
    a.st = h->seq;
    // exact counts for one placement past which a map is the better buy.
    // Fills of 6^9 with limits of 25, 50, 100, 200 and 400: 78.6, 67.9, 66.0,
    // 69.8, 82.0 ms; with 64, 256 and 1000, at maps of twice the time: 7^9
    // 518, 444, 475; 4^11 45, 48, 70.  A quarter of it where tiles make the map
    // (six rounds at 7^9 with 40, 80, 160, 320: 24.8, 24.8, 25.6, 28.9 ms).
    const int evals_map = (int)std::max<long long>(64, std::min<long long>(1024, (long long)h->N / 131072));
    const int evals_tiles = std::max(64, evals_map / 4);
    bool tiled = false;
    int total = 0, vmax = 0;
    long long refreshes = 0, evals = 0, mapped = -1;         // mapped: the words of the last map
    // every refresh that finds a positive gain places at least one word (the
    // first placement of a launch needs no exact count: all bounds are fresh)
    for (int guard = 0; total < room && st.uncov > 0 && guard <= 2 * room + 2; guard++) {
        // bounds: the exact gain map, extracted above a threshold that keeps
        // at most cand_cap candidates.  A word outside the candidates had a
        // gain below the threshold at the refresh (or, when even the map's
        // maximum has more than cand_cap words, the same gain and a higher
        // position): a candidate is placed only while its exact gain is at
        // least the threshold, so it is always a best placement.
        rc = lns_greedy_map(h, st.uncov, mapped < 0 ? -1 : mapped - st.uncov, &tiled);
        if (rc) return rc;
        mapped = st.uncov;
        refreshes++;
        CK(cudaMemsetAsync(h->info, 0x80, offsetof(RefreshInfo, noted)));         // top: a negative number
        CK(cudaMemsetAsync(d_hist, 0, THR_BINS * 4));
        const int *vmax_dev = nullptr;
        if (vmax <= 0) {
            // the first map of the call: its maximum first; later ones are
            // bounded by the last launch's best bound (gains only fall)
            k_lns_max<<<grid_of(h->N), LNS_NT>>>(h->map, h->N, &h->info->top);
            vmax_dev = &h->info->thr;
            CK(cudaMemcpyAsync(&h->info->thr, &h->info->top, 4, cudaMemcpyDeviceToDevice));
        }
        k_lns_tail<<<grid_of(h->N), LNS_NT>>>(h->map, h->N, vmax, vmax_dev, d_hist, &h->info->top);
        k_lns_threshold<<<1, THR_BINS>>>(d_hist, vmax, vmax_dev, (long long)cand_cap, h->info);
        CK(cudaGetLastError());
        rc = extract_launch(h, 1, &h->info->thr, cand_cap, bcount, h->cand, h->bound, nullptr, &h->info->found);
        if (rc) return rc;
        CK(cudaMemsetAsync(h->acc, 0, 4 * (3 * (GREEDY_MAXG + 1) + 1)));
        a.eval_cap = tiled ? evals_tiles : evals_map;
        a.room = room - total;
        a.list = h->list + total;
        a.max_steps = greedy_max_steps(room - total, a.eval_cap);
        void *args[] = {&a};
        CK(cudaLaunchCooperativeKernel((const void *)k_lns_greedy, dim3((unsigned)G), dim3(GREEDY_NT), args, smem, 0));
        CK(cudaMemcpy(&st, h->seq, sizeof st, cudaMemcpyDeviceToHost));
        total += st.placed;
        evals += st.evals;
        vmax = st.best;
        if (st.status == SEQ_GUARD) return COV_ETIMEOUT;
        if (st.status != SEQ_REFRESH || st.placed == 0) break;
    }
    if (total > 0) CK(cudaMemcpy(placed, h->list, (size_t)total * 4, cudaMemcpyDeviceToHost));
    *nplaced = total;
    *uncovered = st.uncov;
    if (stats) { stats[0] = refreshes; stats[1] = evals; }
    return COV_OK;
}

int cov_lns_uncovered(cov_lns *h, int64_t cap, uint32_t *idx, int64_t *found)
{
    if (!h || cap < 0 || (cap > 0 && !idx) || !found) return COV_EINVAL;
    // the indicator of cnt == 0 into the map, then its ordered extraction
    k_lns_indicator<<<grid_of(h->N), LNS_NT>>>(h->cnt, 0, h->N, h->map);
    CK(cudaGetLastError());
    std::vector<int32_t> val((size_t)std::max<int64_t>(std::min<int64_t>(cap, h->N), 1));
    return cov_lns_map_extract(h, 1, cap, idx, val.data(), found);
}

int cov_lns_count(cov_lns *h, int32_t target, int64_t *out)
{
    if (!h || !out || target < 0) return COV_EINVAL;
    CK(cudaMemset(h->d_red, 0, 8));
    k_lns_zero<<<grid_of(h->N), LNS_NT>>>(h->cnt, h->N, target, h->d_red);
    CK(cudaGetLastError());
    unsigned long long z = 0;
    CK(cudaMemcpy(&z, h->d_red, 8, cudaMemcpyDeviceToHost));
    *out = (int64_t)z;
    return COV_OK;
}

int cov_lns_get_cnt(cov_lns *h, uint16_t *out)
{
    if (!h || !out) return COV_EINVAL;
    CK(cudaMemcpy(out, h->cnt, (size_t)h->N * 2, cudaMemcpyDeviceToHost));
    return COV_OK;
}

int cov_lns_get_map(cov_lns *h, int32_t *out)
{
    if (!h || !out) return COV_EINVAL;
    CK(cudaMemcpy(out, h->map, (size_t)h->N * 4, cudaMemcpyDeviceToHost));
    return COV_OK;
}

}  // extern "C"
