// cov_tiles_plan.h -- the tiles of a coverage count (cov_tiles.cuh): their
// limits and their geometry.  Host arithmetic only, so that it compiles
// without CUDA.
#pragma once
#include <cstddef>
#include <cstdint>
#include <algorithm>

#define BT_SMEM_MAX (200 * 1024)    // shared memory of a tile CTA
#define BT_LCH 4096            // codewords of a tile listed at once
#define BT_NT  512             // threads of a tile CTA
#define BT_ITEMS 1024          // ball groups held in shared memory

static inline long long bt_ipow(long long b, int e)
{
    long long r = 1;
    while (e-- > 0) r *= b;
    return r;
}

// digits of a block: the last two (one for words of one digit)
static inline int bt_block_digits(int n) { return n < 2 ? n : 2; }

// ball groups of nm middle digits
static inline long long bt_groups(int q, int nm, int R)
{
    long long g = 0, c = (long long)nm * (nm - 1) / 2;      // C(nm, r) (q-1)^(r-2)
    for (int r = 2; r <= nm && r <= R; r++) {
        g += c;
        c = c * (nm - r) / (r + 1) * (q - 1);
    }
    return g;
}

// dynamic shared memory of a tile CTA: the ball groups, the list, then A0,
// the row and column counters and B
static inline size_t bt_smem_bytes(int q, int n, uint32_t tw)
{
    const size_t nblk = tw / (size_t)bt_ipow(q, bt_block_digits(n));
    return BT_ITEMS * 4 + BT_LCH * 2 + ((size_t)tw + 2 * nblk * q + nblk) * 4;   // bt_layout's words
}

// Tile geometry: the number of low digits with the least estimate, in SM
// cycles, of a tile's prefix tests (about 23 lane-instructions a codeword) and
// words (14 a word) at 64 lanes a cycle and the latency chain of its phases
// (some 6000 cycles, shared by the CTAs resident together).  An SM that works
// at all works a whole tile, so fewer tiles than SMs share nothing: with their
// work counted as spread over the chip, 8^6 R3 with 60000 codewords took eight
// tiles of 8^5 words and 1690 us, and takes 64 and 312; 3^12 R3 M3000 65 and
// 38.  Of 38 cells counted at every number of digits the choice is within 1 %
// of the best in 32 and within 11 % in the rest (before: 1.1 to 5.4 times as
// long in nine).  At most eight high and eight middle digits, which are held
// as 32-bit nibbles.  sms: the device's SMs.
static inline void bt_geom(int q, int n, int R, int M, int sms, int *nh, int *nl)
{
    const int nb = bt_block_digits(n);
    double least = 1e300;
    *nl = -1;
    for (int l = nb > n - 8 ? nb : n - 8; l <= n && l - nb <= 8; l++) {
        const long long tw = bt_ipow(q, l);
        if (tw > (1 << 20) || bt_smem_bytes(q, n, (uint32_t)tw) > BT_SMEM_MAX || bt_groups(q, l - nb, R) > BT_ITEMS)
            break;
        const double tiles = (double)bt_ipow(q, n - l);
        const int res = (int)std::min<size_t>(4, (227 * 1024) / (bt_smem_bytes(q, n, (uint32_t)tw) + 1536));
        const double waves = (double)(long long)((tiles + sms * res - 1) / (sms * res));
        const double cyc = std::max(1.0, tiles / sms) * (M * 23.0 + tw * 14.0) / 64.0 + waves * (6000.0 + M * 0.05);
        if (cyc < least) { least = cyc; *nl = l; }
    }
    *nh = n - *nl;
}

// words within R of a word of n digits
static inline double bt_ball(int q, int n, int R)
{
    double v = 1, c = 1;
    for (int r = 0; r < R && r < n; r++) { c = c * (n - r) / (r + 1) * (q - 1); v += c; }
    return v;
}

// Estimate of counting the balls of m words by tiles, in ps: 1.53 a word of
// the space, and for each of the m 1850 (the chunks of a list, the host's copy)
// and, for each tile of an SM, 650 (its prefix test), 1420 where its ball
// reaches the tile, 1150 a group walked there and 60 a mark, 150 where the
// strides are powers of two and a warp's marks share banks.  Fitted to 548
// counts of 10 to 60,000 words in 71 cells of 2^12 to 8^9 words, R = 1 to 8:
// with 29 us a call, 0.8 to 1.12 times the measured time in eight of ten (0.5
// in the worst, 4^11 R8, where 10,000 words take 8.8 ms).
static inline double bt_count_ps(int q, int n, int R, long long m, int sms)
{
    int nh, nl;
    bt_geom(q, n, R, (int)std::min<long long>(m, 1 << 30), sms, &nh, &nl);
    const double tiles = (double)bt_ipow(q, nh);
    const int nm = nl - bt_block_digits(n);
    double groups = 0, c = 1;
    for (int d = 0; d <= nh && d <= R; d++) {
        groups += c * (double)bt_groups(q, nm, R - d);
        c = c * (nh - d) / (d + 1) * (q - 1);
    }
    const double near = std::min(1.0, bt_ball(q, nh, R) / tiles), marks = bt_ball(q, nm + nh, R) / tiles;
    const double mark = (q & (q - 1)) ? 60.0 : 150.0;
    return 1.53 * tiles * (double)bt_ipow(q, nl) +
           (double)m * (1850.0 + std::max(1.0, tiles / sms) *
                                     (650.0 + 1420.0 * near + 1150.0 * groups / tiles + mark * marks));
}

// The transform of a map or of word counts, ps a word of the space: an axis
// moves R + 1 layers at most (71 cells: 0.7 to 1.2 times the measured time).
static inline double bt_transform_ps(int R) { return 8.8 + 3.3 * R; }

// Whether the counts of m words come from tiles sooner than from the transform
// of their word counts, which takes 13 us of launches and clearing more.
// Measured (us, tiles against transform): 7^8 R1 10,000 words 73, 139, 200,000
// 775, 262; 6^9 R2 3000 74, 198, 30,000 385, 232; 4^11 R4 300 45, 134, 10,000
// 306, 144; 2^16 R5 300 38, 60, 3000 147, 69.
static inline bool bt_tiles_pay(int q, int n, int R, long long m, int sms)
{
    return bt_count_ps(q, n, R, m, sms) < 13e6 + 720.0 * (double)m + bt_transform_ps(R) * (double)bt_ipow(q, n);
}
