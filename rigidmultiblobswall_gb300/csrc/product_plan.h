// How the wall and free-space products split their work, and the scratch that
// takes: rules of sizes and limits alone, with no CUDA in them.
#pragma once
#include <stddef.h>

#include <algorithm>
#include <cmath>

namespace rmw {

constexpr int kPlanTile = 128;        // blobs per tile of the symmetric kernels
constexpr int kSplitMax = 64;         // CTAs per tile pair at most
constexpr double kSplitBytes = 64e6;  // partial sums of a split product (three components): they stay in L2

inline int sym_tiles(int n) { return (n + kPlanTile - 1) / kPlanTile; }

// partial sums of one slot per tile: `comps` (3, or 6 for [U; W]) doubles per blob and tile
inline double sym_slot_bytes(int n, int comps) { return (double)sym_tiles(n) * comps * (double)n * sizeof(double); }

// How many CTAs share the steps of a tile pair.  Below about 4,000 blobs the
// tile pairs alone leave SMs idle (2,048 blobs: 136 of them); the split fills
// the GPU with the symmetric kernel's work per pair where the one-sided kernel
// used to do each pair twice (2,048 blobs: FP64 UF 961 -> 364 us, df64 181 ->
// 70).  With P tile pairs, s CTAs each and a CTA's start and end worth e steps,
// an SM takes (P s / 152 + d)(128 / s + e) step times, d the uneven end of the
// grid: least at s = sqrt(152 * 128 d / (e P)).  Measured by s: df64 UF 2,048
// blobs 8: 72, 16: 74, 32: 81 us; 5,003 blobs 2: 275, 4: 259, 8: 279 us; FP64
// UF 10,752 blobs 1: 8.24, 2: 8.08 ms; FP64 periodic 4,800 blobs 2: 15.2,
// 8: 14.8 ms, which K = 13,000 (df64), 40,000 (FP64) and 160,000 (periodic
// FP64, whose steps are nine times as long) in s = sqrt(K / P) reproduce.
// Where even 64 CTAs per pair are fewer than 16 per SM, the split whose
// busiest SM has least to do (504 blobs FP64: 43, 48 us; 32: 54 us).
inline int sym_split_rule(bool fp64, bool periodic, int n)
{
    const double nt = (double)sym_tiles(n), pairs = 0.5 * nt * (nt + 1);
    int s = 1;
    if (pairs * kSplitMax < 16 * 152.0) {
        const double ends = periodic ? 0.05 : fp64 ? 0.4 : 1.2, fill = fp64 ? 2.0 : 6.0;
        double cost = 0.0;
        for (int c = 1; c <= kSplitMax; ++c) {
            const double t =
                std::max(std::ceil(pairs * c / 152.0), fill) * (std::ceil((double)kPlanTile / c) + ends);
            if (c == 1 || t < 0.99 * cost) {
                cost = t;
                s = c;
            }
        }
    } else {
        s = (int)std::min((double)kSplitMax, std::sqrt((periodic ? 160000.0 : fp64 ? 40000.0 : 13000.0) / pairs) +
                                                     (fp64 ? 0.5 : 0.05));  // whole df64 pairs have constant bounds
    }
    return s;
}

// The rule's split, or the finest below it whose partial sums stay within
// kSplitBytes and `budget` and, with the `packed` bytes of records, within
// the scratch cap (0 = none): a cap that holds the unsplit product never
// costs the symmetric kernel.
inline int sym_split(bool fp64, bool periodic, int n, int comps, double packed, double budget, double cap)
{
    const double slot = sym_slot_bytes(n, comps), most = std::min(kSplitBytes * comps / 3, budget);
    int s = sym_split_rule(fp64, periodic, n);
    while (s > 1 && (slot * s > most || (cap > 0 && packed + slot * s > cap))) --s;
    return std::max(1, s);
}

// Partial sums that a symmetric product's buffer has room for: at least what
// any smaller product takes, whose split may be finer (df64: 22 MB at 10,752
// blobs, 38 MB at 10,000), so that a buffer that served n blobs serves every
// smaller n, also where it must not grow (a stream capture).
inline double sym_reserve_bytes(int n, int comps)
{
    const double slot = sym_slot_bytes(n, comps);
    return std::max(slot, std::min(kSplitBytes * comps / 3, kSplitMax * slot));
}

// The one-sided kernels' source chunks: enough CTAs to fill the 152 SMs
// several times over, at least 256 sources each.
inline int coarse_chunks(int n)
{
    const int tiles = sym_tiles(n);
    const int s = std::min((152 * 8 + tiles - 1) / tiles, std::max(1, n / 256));
    return std::max(1, std::min(s, kSplitMax));
}

// The same in FP64 and df64 (periodic products, fewer than 256 blobs): the
// split whose busiest SM has the least to do, counting a tile's staging as two
// sources; an SM needs about two FP64 or four df64 CTAs to keep its pipe busy.
// coarse_chunks left 1,500 periodic blobs on 60 CTAs.  Finer than that only
// while the partial sums stay within kSplitBytes and, with the packed records,
// within the scratch cap (0 = none).
inline int fine_chunks(bool fp64, int n, double packed, double cap)
{
    const int base = coarse_chunks(n), tiles = sym_tiles(n), fill = fp64 ? 2 : 4;
    const double one = 3.0 * (double)n * sizeof(double);
    int best = base;
    long long cost = -1;
    for (int c = 1; c <= kSplitMax && c <= std::max(base, n / 8); ++c) {
        if (c > base && (one * c > kSplitBytes || (cap > 0 && packed + one * c > cap))) break;
        const long long ctas = ((long long)tiles * c + 151) / 152;
        const long long t = std::max<long long>(ctas, fill) * ((n + c - 1) / c + 2);
        if (cost < 0 || t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

// as sym_reserve_bytes, for fine_chunks
inline double fine_reserve_bytes(int n)
{
    const double one = 3.0 * (double)n * sizeof(double);
    return std::max(one * coarse_chunks(n), std::min(kSplitBytes, kSplitMax * one));
}

}  // namespace rmw
