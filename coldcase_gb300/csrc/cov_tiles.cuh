// cov_tiles.cuh -- coverage counting by tiles of the word space, shared by
// the engine's state build (cov_engine.cu) and the verifier's multiplicity
// count (cov_verify.cu).
//
// A tile is the q^nl consecutive words that share their first nh digits.
// Every codeword within distance R of the tile's prefix adds to it the ball
// of radius rho = R - d(prefix) on the low digits; the tile is worked in
// shared memory, so that the M*|B| increments of the reference's rebuild
// (covsearch2e.c:958-967, M x ball_apply) are shared-memory atomics and the
// counts reach HBM once.
//
// Of the low digits only the middle ones (all but the last two) are walked
// word by word.  A block is the q x q words that share all digits but the
// last two; at a block r middle digits away from the codeword, the remaining
// radius sigma = rho - r decides what the ball covers there: the codeword's
// own last two digits (0), their row and column (1) or the whole block (>= 2).
// A mark is one add to the word's counter A0 (0), one to the block's counter B
// (>= 2), or (1) one to the row's counter, one to the column's and one
// subtraction from the word that lies in both; afterwards each word collects
// A0 + row + column + B.  A codeword costs V(n-2, R) marks instead of V(n, R):
// 53,719 for 182,791 at q7 n9 R4, 7,560 of them of the three-fold kind.  The
// sums are of 32-bit words mod 2^32, so they serve any added value (the engine
// adds 1 + (id << 16)).
#pragma once
#include <cstdint>
#include <vector>
#include <algorithm>
#include "cov_common.cuh"
#include "cov_tiles_plan.h"

// The ball of radius <= min(R, nl) on the digits nh..n-1 (nl of them) as groups: a
// group fixes the values of the first r-1 positions of an r-subset (nibble
// j of items[] is the value index at position j plus 1, 0 where the centre's
// digit stays) and runs over the q-1 values of its last position last[] (r =
// 0: the centre alone, last = 0xff).  gcum[r] groups have radius <= r.
static inline std::vector<uint64_t> bt_items_h(int q, int n, int R, int nh, uint32_t *gcum,
                                               std::vector<uint8_t> &last)
{
    const int nl = n - nh, rmax = std::min(R, nl);
    std::vector<uint64_t> out;
    last.clear();
    out.push_back(0);
    last.push_back(0xff);
    gcum[0] = 1;
    for (int r = 1; r <= rmax; r++) {
        std::vector<int> sub(r);
        for (int k = 0; k < r; k++) sub[k] = k;
        while (true) {
            std::vector<int> dig(r - 1, 0);
            while (true) {
                uint64_t sp = 0;
                for (int k = 0; k < r - 1; k++) sp |= (uint64_t)(dig[k] + 1) << (4 * (nh + sub[k]));
                out.push_back(sp);
                last.push_back((uint8_t)(nh + sub[r - 1]));
                int k = r - 2;
                while (k >= 0 && dig[k] == q - 2) dig[k--] = 0;
                if (k < 0) break;
                dig[k]++;
            }
            int k = r - 1;
            while (k >= 0 && sub[k] == nl - r + k) k--;
            if (k < 0) break;
            sub[k]++;
            for (int m = k + 1; m < r; m++) sub[m] = sub[m - 1] + 1;
        }
        gcum[r] = (uint32_t)out.size();
    }
    return out;
}

// What a tile needs of each codeword, made once per call by k_bt_records:
// the high digits as nibbles, and {middle digits as nibbles, (block of the
// middle digits << 8) | word in the block}.
struct BtCode {
    const uint32_t *hi;
    const uint2 *mid;
};
#define BT_REC_BYTES 12        // bytes of one codeword's records

template <class Digit>
__device__ __forceinline__ void bt_record(int i, int q, int n, int nh, int nl, uint2 *mid, uint32_t *hi, Digit digit)
{
    const int nb = n < 2 ? n : 2;
    uint32_t h = 0, m = 0, z = 0, y = 0;
    for (int j = 0; j < nh; j++) h |= digit(j) << (4 * j);
    for (int j = nh; j < n - nb; j++) { m |= digit(j) << (4 * (j - nh)); z = z * (uint32_t)q + digit(j); }
    for (int j = n - nb; j < n; j++) y = y * (uint32_t)q + digit(j);
    hi[i] = h;
    mid[i] = make_uint2(m, (z << 8) | y);
}

static __global__ void k_bt_records(const uint64_t *__restrict__ code, int M, int q, int n, int nh, int nl, uint2 *mid,
                                    uint32_t *hi)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const uint64_t pc = code[i];
        bt_record(i, q, n, nh, nl, mid, hi, [&](int j) { return (uint32_t)cov_nib(pc, j); });
    }
}

// records of M packed codewords into rec (M * BT_REC_BYTES bytes, 8-byte aligned)
static inline BtCode bt_records(const uint64_t *d_code, int M, int q, int n, int nh, int nl, void *rec, cudaStream_t st)
{
    uint2 *mid = (uint2 *)rec;
    uint32_t *hi = (uint32_t *)(mid + M);
    if (M > 0) k_bt_records<<<std::min(1024, (M + 127) / 128), 128, 0, st>>>(d_code, M, q, n, nh, nl, mid, hi);
    return BtCode{hi, mid};
}

// the tile's arrays as word offsets in dynamic shared memory
struct BtTile {
    uint32_t list, a0, row, col, b, words;      // (item at 0); list: 16-bit entries
};

__host__ __device__ __forceinline__ BtTile bt_layout(int q, int n, uint32_t tw)
{
    BtTile t;
    const uint32_t nblk = tw / (uint32_t)(n < 2 ? q : q * q);
    t.list = BT_ITEMS;
    t.a0 = t.list + BT_LCH / 2;
    t.row = t.a0 + tw;
    t.col = t.row + nblk * (uint32_t)q;
    t.b = t.col + nblk * (uint32_t)q;
    t.words = t.b + nblk;
    return t;
}

// alphabet sizes with their own tile-marking kernels (others run Q = 0)
#define BT_Q_LIST(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)

__device__ __forceinline__ int bt_dist8(uint32_t a, uint32_t b)
{
    uint32_t x = a ^ b;
    x |= x >> 1;
    x |= x >> 2;
    return __popc(x & 0x11111111u);
}

__device__ __forceinline__ void bt_add(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Fill the tile numbered `index`: the balls of codewords 0..M-1 intersecting
// it, inc(id) added per covered word; the sums stand in sm[tl.a0 ..] when it
// returns (sm: the kernel's dynamic shared memory, laid out by bt_layout).
// vcum_ is bt_vcum_h's.  Q > 0: the alphabet size at compile time; Q = 0:
// any q and words of one digit.  Every thread of the CTA (BT_NT) calls it.
//
// Bound by the latency of its phases and by issue: at 7^9 with 1500 codewords
// 137 us (two CTAs an SM, 59 % of the issue slots), 65 us of it with 8
// codewords.  Marking every ball word in a tile of its own digits took 276 us
// (8^10, 2549 codewords: 9.2 -> 3.1 ms); tiles of 7^4, four CTAs an SM: 512 us,
// because seven times the tiles test every prefix and meet at every barrier.
template <int Q, class Inc>
__device__ __forceinline__ void bt_mark_tile(uint32_t *sm, const BtTile tl, uint32_t index, int q_, int n, int R, int M,
                                             const BtCode code, int nh, int nl, const uint32_t *vcum_, Inc inc)
{
    constexpr int KEEP = BT_LCH / BT_NT;
    const int q = Q > 0 ? Q : q_;
    const int nb = Q > 0 || n >= 2 ? 2 : 1, nm = nl - nb;     // digits of a block, middle digits
    __shared__ uint32_t pz[8];                      // block strides of the middle digits
    __shared__ uint32_t vcum[COV_MAXN + 2];
    __shared__ int seg[(COV_MAXN + 1) * 9];
    __shared__ int gcnt[COV_MAXN + 2], gpos[COV_MAXN + 2], gfill[COV_MAXN + 2];
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    uint16_t *const list = reinterpret_cast<uint16_t *>(sm + tl.list);
    if (threadIdx.x < 8) {
        uint32_t p = 1;
        for (int j = nm - 1; j > (int)threadIdx.x; j--) p *= (uint32_t)q;
        pz[threadIdx.x] = p;
    }
#pragma unroll
    for (int r = 0; r < COV_MAXN + 2; r++)
        if (threadIdx.x == 0) vcum[r] = vcum_[r];
    uint32_t hp = 0;
    for (int j = nh - 1; j >= 0; --j) { hp |= (index % (uint32_t)q) << (4 * j); index /= (uint32_t)q; }
    const uint32_t blk = (uint32_t)(nb == 2 ? q * q : q);
    uint32_t nblk = 1;
    for (int j = 0; j < nm; j++) nblk *= (uint32_t)q;
    const int rmax = min(R, nm);
    {
        // a0, row, col and b in a row, from a 16-byte boundary
        const uint32_t words = tl.words - tl.a0;
        uint4 *z4 = reinterpret_cast<uint4 *>(sm + tl.a0);
        for (uint32_t x = threadIdx.x; x < words / 4; x += BT_NT) z4[x] = make_uint4(0, 0, 0, 0);
        if (threadIdx.x < (words & 3u)) sm[tl.a0 + (words & ~3u) + threadIdx.x] = 0;
    }
    __syncthreads();
    // the groups: an r-subset of the middle digits (r >= 2) with the value
    // indices of its first r - 2 positions, plus 1, as nibbles, and 15 at its
    // last two positions
    for (uint32_t i = threadIdx.x; i < vcum[rmax]; i += BT_NT) {
        int r = 2;
        while (i >= vcum[r]) r++;
        uint32_t combos = 1;
        for (int k = 2; k < r; k++) combos *= (uint32_t)(q - 1);
        uint32_t v = i - vcum[r - 1], nth = v / combos, set = 0;
        v -= nth * combos;
        for (set = 0;; set++)
            if (__popc(set) == r && nth-- == 0) break;
        uint32_t sp = 0, rest = set;
        for (int k = 0; k < r; k++) {
            const int j = __ffs((int)rest) - 1;
            rest &= rest - 1;
            sp |= (k < r - 2 ? v % (uint32_t)(q - 1) + 1u : 15u) << (4 * j);
            if (k < r - 2) v /= (uint32_t)(q - 1);
        }
        sm[i] = sp;
    }
    const int lane = threadIdx.x & 31;
    for (int m0 = 0; m0 < M; m0 += BT_LCH) {
        const int m1 = min(M, m0 + BT_LCH);
        if ((int)threadIdx.x <= R) gcnt[threadIdx.x] = 0;
        __syncthreads();
        // codewords per remaining radius, then their list grouped by it; the
        // lanes of a warp that share a radius go together
        int rho[KEEP];
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const int k = m0 + u * BT_NT + (int)threadIdx.x;
            rho[u] = -1;
            if (m0 + u * BT_NT < m1) {
                if (k < m1) rho[u] = R - bt_dist8(__ldg(&code.hi[k]), hp);
                unsigned left = __ballot_sync(0xffffffffu, rho[u] >= 0);
                while (left) {
                    const int r = __shfl_sync(0xffffffffu, rho[u], __ffs(left) - 1);
                    const unsigned m = __ballot_sync(0xffffffffu, rho[u] == r);
                    if (lane == 0) atomicAdd(&gcnt[r], __popc(m));
                    left &= ~m;
                }
            }
        }
        __syncthreads();
        // Segments (rho, r): the codewords with remaining radius rho and the
        // groups of radius r on the middle digits, so that sigma and the
        // digits of a group are the same for a whole warp (lanes of different
        // kinds would run each other's marks).  r = 0: the centre alone
        // (rho = 0); r = 1: the centre and every single digit, one lane a
        // codeword; r >= 2: a group fixes all digits but its last two, so that
        // the walk to it is shared by (q-1)^2 marks.  A warp takes 32
        // (codeword, group) pairs of one segment at a time.
        const int nseg = (R + 1) * (rmax + 1);
        if (threadIdx.x < 32) {
            int run = 0;
            for (int s0 = 0; s0 < nseg; s0 += 32) {
                const int s = s0 + lane;
                int c = 0;
                if (s < nseg) {
                    const int h = s / (rmax + 1), r = s - h * (rmax + 1);
                    const int groups = r >= 2 ? (int)(vcum[r] - vcum[r - 1]) : (r == min(1, min(h, rmax)) ? 1 : 0);
                    c = r <= h ? (gcnt[h] * groups + 31) / 32 : 0;
                }
                int x = c;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (s < nseg) seg[s] = run + x;              // chunks up to and with segment s
                run += __shfl_sync(0xffffffffu, x, 31);
            }
        } else if (threadIdx.x == 32) {
            int acc = 0;
            for (int r = 0; r <= R; r++) { gpos[r] = acc; gfill[r] = acc; acc += gcnt[r]; }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            if (m0 + u * BT_NT < m1) {
                unsigned left = __ballot_sync(0xffffffffu, rho[u] >= 0);
                while (left) {
                    const int r = __shfl_sync(0xffffffffu, rho[u], __ffs(left) - 1);
                    const unsigned m = __ballot_sync(0xffffffffu, rho[u] == r);
                    int at = 0;
                    if (lane == 0) at = atomicAdd(&gfill[r], __popc(m));
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (rho[u] == r)
                        list[at + __popc(m & ((1u << lane) - 1))] = (uint16_t)(u * BT_NT + (int)threadIdx.x);
                    left &= ~m;
                }
            }
        }
        __syncthreads();
        const int chunks = seg[nseg - 1];
        int sg = 0, h = 0, r = 0;                            // the warp's segment, its rho and radius
        for (int ch = threadIdx.x >> 5; ch < chunks; ch += BT_NT / 32) {
            while (seg[sg] <= ch) {
                sg++;
                if (++r > rmax) { r = 0; h++; }
            }
            const uint32_t g0 = r >= 2 ? vcum[r - 1] : 0u, V = r >= 2 ? vcum[r] - g0 : 1u;
            const uint32_t t = (uint32_t)(ch - (sg ? seg[sg - 1] : 0)) * 32u + (uint32_t)lane;
            if (t >= (uint32_t)gcnt[h] * V) continue;
            uint32_t kk = t, it = 0;
            if (V > 1) {
                // t / V; t < BT_LCH * BT_ITEMS < 2^24, so one correction makes it exact
                kk = (uint32_t)((float)t * __fdividef(1.0f, (float)V));
                int rem = (int)t - (int)(kk * V);
                if (rem < 0) { kk--; rem += (int)V; } else if (rem >= (int)V) { kk++; rem -= (int)V; }
                it = (uint32_t)rem;
            }
            const int id = m0 + list[gpos[h] + (int)kk];
            const uint2 c = __ldg(&code.mid[id]);
            const uint32_t add = inc((uint32_t)id), y = c.y & 255u;
            const uint32_t yr = y / (uint32_t)q, yc = y - yr * (uint32_t)q;
            uint32_t z = c.y >> 8;
            // the mark of block zz at remaining radius sigma, and those of
            // the q - 1 other values of a middle digit of stride step there,
            // cyclically from the centre's, which lies `up` below the wrap
            auto mark_one = [&](uint32_t zz, int sigma) {
                if (sigma >= nb) {
                    bt_add(sbase + 4u * (tl.b + zz), add);
                } else if (sigma == 0) {
                    bt_add(sbase + 4u * (tl.a0 + zz * blk + y), add);
                } else {
                    bt_add(sbase + 4u * (tl.row + zz * (uint32_t)q + yr), add);
                    bt_add(sbase + 4u * (tl.col + zz * (uint32_t)q + yc), add);
                    bt_add(sbase + 4u * (tl.a0 + zz * blk + y), 0u - add);
                }
            };
            auto mark_line = [&](uint32_t zz, uint32_t step, int up, int sigma) {
                if (sigma >= nb || sigma == 0) {
                    uint32_t at = sbase + 4u * (sigma ? tl.b + zz : tl.a0 + zz * blk + y);
                    const uint32_t st = 4u * (sigma ? step : step * blk), wrap = st * (uint32_t)q;
#pragma unroll
                    for (int v = 0; v < (Q > 0 ? Q : COV_MAXQ) - 1; v++) {
                        if (Q == 0 && v >= q - 1) break;
                        at += st;
                        if (v == up) at -= wrap;
                        bt_add(at, add);
                    }
                } else {
                    uint32_t at = sbase + 4u * (tl.a0 + zz * blk + y), ar = sbase + 4u * (tl.row + zz * (uint32_t)q + yr);
                    const uint32_t co = 4u * (tl.col - tl.row + yc - yr);
                    const uint32_t sr = 4u * step * (uint32_t)q, sa = sr * (uint32_t)q;
#pragma unroll
                    for (int v = 0; v < (Q > 0 ? Q : COV_MAXQ) - 1; v++) {
                        if (Q == 0 && v >= q - 1) break;
                        at += sa;
                        ar += sr;
                        if (v == up) { at -= sa * (uint32_t)q; ar -= sr * (uint32_t)q; }
                        bt_add(ar, add);
                        bt_add(ar + co, add);
                        bt_add(at, 0u - add);
                    }
                }
            };
            if (r < 2) {
                mark_one(z, h);
                if (r)
                    for (int j = 0; j < nm; j++) mark_line(z, pz[j], q - 1 - (int)((c.x >> (4 * j)) & 15u), h - 1);
            } else {
                // a group: a nibble is the value index at its middle digit
                // plus 1, but for the two highest
                uint32_t sp = sm[g0 + it];
                for (int k = 2; k < r; k++) {
                    const int j4 = (__ffs((int)sp) - 1) & ~3;
                    const int dig = (int)((sp >> j4) & 15u) - 1, cj = (int)((c.x >> j4) & 15u);
                    sp &= ~(15u << j4);
                    z += (uint32_t)((dig + (dig >= cj) - cj) * (int)pz[j4 >> 2]);
                }
                const int ja = (__ffs((int)sp) - 1) >> 2, jb = (31 - __clz((int)sp)) >> 2;
                const uint32_t sa = pz[ja], sb = pz[jb];
                const int ua = q - 1 - (int)((c.x >> (4 * ja)) & 15u), ub = q - 1 - (int)((c.x >> (4 * jb)) & 15u);
                for (int v = 0; v < q - 1; v++) {
                    z += sa;
                    if (v == ua) z -= sa * (uint32_t)q;
                    mark_line(z, sb, ub, h - r);
                }
            }
        }
        __syncthreads();
    }
    // collect, a thread per row of a block; q = 8 rows start at different
    // columns, or eight lanes would meet in a bank
    const uint32_t qr = nb == 2 ? (uint32_t)q : 1u;         // rows of a block
    for (uint32_t l = threadIdx.x; l < nblk * qr; l += BT_NT) {
        const uint32_t z = l / qr;
        const uint32_t s = sm[tl.b + z] + (nb == 2 ? sm[tl.row + l] : 0u);
        const uint32_t *col = sm + tl.col + z * (uint32_t)q;
        uint32_t *a0 = sm + tl.a0 + l * (uint32_t)q;
        if constexpr (Q > 0) {
#pragma unroll
            for (int y = 0; y < Q; y++) {
                const int yy = Q == 8 ? ((y + (int)(l >> 2)) & 7) : y;
                a0[yy] += s + col[yy];
            }
        } else {
            for (int y = 0; y < q; y++) a0[y] += s + (nb == 2 ? col[y] : 0u);
        }
    }
    __syncthreads();
}

// vcum[r]: the groups of radius 2 .. r on the middle digits of a tile
static inline void bt_vcum_h(int q, int n, int R, int nl, uint32_t *vcum)
{
    const int nm = nl - bt_block_digits(n);
    long long c = (long long)nm * (nm - 1) / 2;             // C(nm, r) (q-1)^(r-2)
    vcum[0] = vcum[1] = 0;
    for (int r = 2; r <= COV_MAXN + 1; r++) {
        const bool in = r <= nm && r <= R;
        vcum[r] = vcum[r - 1] + (in ? (uint32_t)c : 0u);
        if (in) c = c * (nm - r) / (r + 1) * (q - 1);
    }
}

// cov_verify.cu: the saturated coverage counts of the m listed words (device
// word indices below q^n) into cnt; rec: m * BT_REC_BYTES bytes, 8-byte aligned
int cov_count_words(int q, int n, int R, const uint32_t *d_idx, int m, uint16_t *cnt, uint2 *rec, cudaStream_t st);
// the same counts unsaturated into map, or (subtract) off it
int cov_count_words_map(int q, int n, int R, const uint32_t *d_idx, int m, int32_t *map, int subtract, uint2 *rec,
                        cudaStream_t st);
